"""Host side of the GEMM over a cluster: blocks that fit one SM together never wait for one another's tensor memory."""
import itertools
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SM_SMEM, SM_COLUMNS, RESERVED = 228 * 1024, 512, 1024     # of sm_100; the reserve is a block's


def plans(tmp_path, *args):
    exe = str(tmp_path / "plans")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "dyninfer_b200", "csrc"),
                           os.path.join(ROOT, "tests", "gemm_cluster_plans.cpp"), "-o", exe])
    return subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True).stdout.splitlines()


@pytest.mark.parametrize("sms", [148, 132])
def test_plans_that_fit_an_sm_together_fit_its_tensor_memory(tmp_path, sms):
    """A block waits for its columns and then for its cluster, so two plans that shared an SM without room for both their
    columns could wait for one another across two SMs. By their smallest shared memory, any number of blocks of any kinds."""
    kinds = [tuple(map(int, line.split())) for line in plans(tmp_path, sms)]
    assert {k[0] for k in kinds} == {256, 512}              # both kinds are met
    for columns, least, largest, count, holds in kinds:
        assert count > 1000 and holds and least <= largest <= 222 * 1024
    for n in range(2, 6):
        for together in itertools.combinations_with_replacement(kinds, n):
            if sum(k[1] + RESERVED for k in together) <= SM_SMEM:
                assert sum(k[0] for k in together) <= SM_COLUMNS, together


WORDS = {"gguf.q4_0": 36, "gguf.q4_1": 40, "gguf.q8_0": 68, "gguf.q4_k": 36, "gguf.q5_k": 44, "mlx.affine.u4": 32}


def test_products_that_the_gpu_tests_mean_go_over_a_cluster(tmp_path):
    """The dispatch's own rule at the sizes of test_linear_rows_over_a_cluster (of which K = 256 is too little and 6400 too much) and of
    test_linear_encodings_over_a_cluster, all of whose products it has to take."""
    sizes = [(33, 130, 256), (48, 127, 768), (49, 1000, 2560), (64, 257, 3072), (47, 2049, 1792), (64, 6000, 1024), (40, 128, 6144),
             (64, 129, 6400), (65, 1024, 2048), (128, 257, 1536), (100, 2048, 2048), (127, 1000, 3072)]
    for words in (32, 36, 40, 68):
        got = plans(tmp_path, 148, *(v for m, n, k in sizes for v in (m, n, k, words)))
        assert [int(ck) > 0 for ck in got] == [k not in (256, 6400) for _, _, k in sizes], (words, got)
    from test_gpu_paths import CLUSTER_PRODUCTS
    got = plans(tmp_path, 148, *(v for enc, m, n, k, _, _ in CLUSTER_PRODUCTS for v in (m, n, k, WORDS[enc])))
    assert all(int(ck) >= 2 for ck in got), got
