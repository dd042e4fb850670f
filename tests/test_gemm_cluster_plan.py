"""Host side of the GEMM over a cluster: blocks that fit one SM together never wait for one another's tensor memory."""
import itertools
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SM_SMEM, SM_COLUMNS, RESERVED = 228 * 1024, 512, 1024     # of sm_100; the reserve is a block's


@pytest.mark.parametrize("sms", [148, 132])
def test_plans_that_fit_an_sm_together_fit_its_tensor_memory(tmp_path, sms):
    """A block waits for its columns and then for its cluster, so two plans that shared an SM without room for both their
    columns could wait for one another across two SMs. By their smallest shared memory, any number of blocks of any kinds."""
    exe = str(tmp_path / "plans")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "dyninfer_b200", "csrc"),
                           os.path.join(ROOT, "tests", "gemm_cluster_plans.cpp"), "-o", exe])
    lines = subprocess.run([exe, str(sms)], check=True, capture_output=True, text=True).stdout.splitlines()
    kinds = [tuple(map(int, line.split())) for line in lines]
    assert {k[0] for k in kinds} == {256, 512}              # both kinds are met
    for columns, least, largest, count, holds in kinds:
        assert count > 1000 and holds and least <= largest <= 222 * 1024
    for n in range(2, 6):
        for together in itertools.combinations_with_replacement(kinds, n):
            if sum(k[1] + RESERVED for k in together) <= SM_SMEM:
                assert sum(k[0] for k in together) <= SM_COLUMNS, together
