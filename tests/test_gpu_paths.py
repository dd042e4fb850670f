"""Kernel variants at the sizes where their dispatch or their tiling changes, against the CPU oracle."""
import numpy as np
import pytest

import helpers
from dyninfer_b200 import synth
from dyninfer_b200.runtime import ModelLoader, SessionConfig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("s,start,nh,nkv,mag", [(32, 0, 2, 2, 1.0), (100, 37, 4, 2, 1.0), (130, 500, 4, 1, 1e6),
                                                (65, 31, 40, 8, 1e-12)])
def test_attention_prefill_f32_cache(native_lib, oracle, s, start, nh, nkv, mag):
    """32 or more consecutive rows on an f32 cache (f16 pairs on the tensor cores): f32 accuracy, ragged row
    blocks, rows that start inside a key step, values far outside the f16 range with a scale per tile."""
    from dyninfer_b200 import ops
    d, cap = 128, 768
    rng = np.random.default_rng(s + start)
    q = (rng.normal(size=(s, nh, d)) / mag).astype(np.float32)
    kc = (rng.normal(size=(nkv, cap, d)) * mag).astype(np.float32)
    vc = (rng.normal(size=(nkv, cap, d)) * mag * np.exp2(rng.integers(0, 12, size=(1, cap // 64, 1))).repeat(64, 1)).astype(np.float32)
    kc[:, start + s:] = np.nan                 # never-written rows must not leak into the result
    vc[:, start + s:] = np.nan
    got = ops.attention(torch.from_numpy(q).cuda(), torch.from_numpy(kc).cuda(), torch.from_numpy(vc).cuda(), start).cpu().numpy()
    want = oracle.attention(q, np.nan_to_num(kc), np.nan_to_num(vc), start, s)
    assert np.isfinite(got).all()
    assert helpers.rel_err(got, want) < 2e-5


SKINNY = ["gguf.q4_0", "gguf.q4_1", "gguf.q8_0", "gguf.q6_k", "gguf.q4_k", "mlx.affine.u4", "plain.bf16", "plain.f16"]


@pytest.mark.parametrize("enc", SKINNY)
@pytest.mark.parametrize("m,n,k", [(5, 40, 512), (8, 1000, 3072), (9, 33, 5120), (16, 130, 1024), (17, 1024, 2048),
                                   (33, 513, 1536), (64, 4096, 1024), (64, 48, 12800)])
def test_linear_few_rows(native_lib, oracle, enc, m, n, k):
    """5 to 64 activation rows: ragged rows and tiles, row groups of 8 that are not full, K split over warps and
    over the CTAs of a cluster; a row of zeros and one far outside the f16 range."""
    from dyninfer_b200 import ops
    from test_gpu_ops import make_pair
    dw, ow = make_pair(oracle, enc, n, k, seed=n + m)
    x = np.random.default_rng(m).normal(size=(m, k)).astype(np.float32)
    x[1] = 0.0
    x[2] *= 1e7
    got = ops.linear(dw, torch.from_numpy(x).cuda()).cpu().numpy()
    want = oracle.linear(ow, x, fast=True)
    assert np.isfinite(got).all()
    for r in (0, 2, m - 1):
        assert helpers.rel_err(got[r], want[r]) < 1e-3
    assert not got[1].any()
    others = np.delete(np.arange(m), 2)
    assert helpers.rel_err(got[others], want[others]) < (1e-5 if enc.startswith("plain") and m <= 16 else 1e-3)
    if m > 8:
        xb = torch.from_numpy(x).to(torch.bfloat16)
        got = ops.linear(dw, xb.cuda()).cpu().numpy()
        assert helpers.rel_err(got[others], oracle.linear(ow, xb.float().numpy(), fast=True)[others]) < 1e-3


@pytest.mark.parametrize("enc", ["gguf.q4_0", "gguf.q4_1", "gguf.q8_0", "gguf.q6_k", "gguf.q4_k", "mlx.affine.u4"])
@pytest.mark.parametrize("m,n,k", [(1, 17, 512), (2, 100, 1024), (3, 1000, 3072), (4, 40, 25600), (7, 513, 2048),
                                   (8, 33, 12800)])
def test_linear_exact_rows(native_lib, oracle, enc, m, n, k):
    """1 to 4 f32 rows and 1 to 8 bf16 rows keep the weights exact: f32 accuracy, ragged tiles, K split over warps and
    clusters, rows of zeros, of huge and of mixed magnitude."""
    from dyninfer_b200 import ops
    from test_gpu_ops import make_pair
    dw, ow = make_pair(oracle, enc, n, k, seed=n + m)
    x = np.random.default_rng(m).normal(size=(m, k)).astype(np.float32)
    x[0, ::5] *= 1e-4
    if m > 1:
        x[1] = 0.0
    if m > 2:
        x[2] *= 1e9
    xb = torch.from_numpy(x).to(torch.bfloat16)
    for t in ([torch.from_numpy(x), xb] if m <= 4 else [xb]):
        got = ops.linear(dw, t.cuda()).cpu().numpy()
        want = oracle.linear(ow, t.float().numpy(), fast=True)
        for r in range(m):
            assert helpers.rel_err(got[r], want[r]) < 2e-5 if r != 1 else not got[r].any()


@pytest.mark.gpu
@pytest.mark.parametrize("keys", [63, 64, 128, 129, 575, 1030])
def test_persistent_attention_slices(native_lib, tmp_path, keys):
    """One, two, three and the most slices of a head's keys, merged by the head's own blocks, against the operator path."""
    path = synth.write_qwen3_gguf(str(tmp_path / "q.gguf"), synth.SMALL_D128, seed=5)
    prompt = np.random.default_rng(keys).integers(0, 512, size=keys).tolist()
    got = []
    for kernel in ("persistent", "graph"):
        model = ModelLoader().load(path, max_kv=1152, kv_dtype="bf16", chunk_size=128, decode_kernel=kernel)
        with model.create_session(SessionConfig(max_sequence_length=1152)) as s:
            assert s.uses_persistent_kernel() == (kernel == "persistent")
            s.prefill(prompt)
            got.append(np.stack([s.decode(t).values.copy() for t in (7, 11)]))
    assert np.abs(got[0] - got[1]).max() <= 1e-3


@pytest.mark.parametrize("enc", ["gguf.q4_0", "gguf.q4_1", "gguf.q8_0", "gguf.q4_k", "gguf.q5_k", "mlx.affine.u4"])
@pytest.mark.parametrize("m,n,k", [(65, 40, 256), (70, 129, 5120), (100, 19000, 512), (129, 640, 4096), (257, 257, 1024),
                                   (600, 4096, 768)])
def test_linear_many_rows(native_lib, oracle, enc, m, n, k):
    """Ragged rows and tiles, one and several tiles of activation rows, tiles finished by one block and by several, more
    tiles than blocks; rows of zeros and one far outside the f16 range; the same bits from call to call."""
    from dyninfer_b200 import ops
    from test_gpu_ops import make_pair
    dw, ow = make_pair(oracle, enc, n, k, seed=n + m)
    x = np.random.default_rng(m).normal(size=(m, k)).astype(np.float32)
    x[1] = 0.0
    x[2] *= 1e7
    rows = [0, 2, 3, 63, 64, m // 2, m - 2, m - 1]
    for t in (torch.from_numpy(x), torch.from_numpy(x).to(torch.bfloat16)):
        dev = t.cuda()
        first = ops.linear(dw, dev)
        got = first.cpu().numpy()
        want = oracle.linear(ow, t.float().numpy()[rows], fast=True)
        assert np.isfinite(got).all() and not got[1].any()
        for i, r in enumerate(rows):
            assert helpers.rel_err(got[r], want[i]) < 1e-3
        assert torch.equal(first, ops.linear(dw, dev))


@pytest.mark.parametrize("slots", [5, 33, 64])
def test_batched_attention_few_and_many_rows(native_lib, tmp_path, slots):
    """Slices merged over a cluster (up to a block per SM) and through memory (more), against one sequence at a time."""
    cfg = dict(synth.SMALL_D128, heads=8, kv_heads=4)
    path = synth.write_qwen3_gguf(str(tmp_path / "q.gguf"), cfg, seed=9)
    model = ModelLoader().load(path, max_kv=640, kv_dtype="bf16", chunk_size=64, decode_kernel="graph")
    rng = np.random.default_rng(slots)
    prompts = [rng.integers(0, 512, size=int(n)).tolist() for n in rng.integers(1, 600, size=slots)]
    with model.create_batched_session(SessionConfig(max_sequence_length=640, batch_size=slots)) as s:
        for b, p in enumerate(prompts):
            s.prefill_slot(b, p, want_logits=True)
        s.step({b: 7 for b in range(slots)})
        _, logits = s.step({b: 11 for b in range(slots)}, want_logits=True)
        logits = np.array([logits[b] for b in (0, 1, slots - 1)])
    for i, b in enumerate((0, 1, slots - 1)):
        with model.create_session(SessionConfig(max_sequence_length=640)) as s:
            s.prefill(prompts[b])
            s.decode(7)
            want = s.decode(11).values
        assert np.abs(logits[i] - want).max() <= 1e-2 and helpers.cosine(logits[i], want) >= 0.9999


@pytest.mark.parametrize("enc", ["gguf.q4_0", "gguf.q8_0", "gguf.q6_k", "mlx.affine.u4", "plain.bf16", "plain.f16"])
@pytest.mark.parametrize("m", [1, 4, 5, 16, 40, 100])
def test_linear_rows_at_the_ends_of_the_range(native_lib, oracle, enc, m):
    """Rows are scaled into the f16 range by a power of two: it stays finite for rows of 1e-36 and, where more than four
    rows are scaled by it alone, for a row that holds the largest f32."""
    from dyninfer_b200 import ops
    from test_gpu_ops import make_pair
    n, k = 96, 512
    dw, ow = make_pair(oracle, enc, n, k, seed=m)
    x = np.random.default_rng(m).normal(size=(m, k)).astype(np.float32)
    x[0] *= 1e-36
    if m > 4:
        x[1] = 0.0
        x[1, 77] = 3.4e38
    got = ops.linear(dw, torch.from_numpy(x).cuda()).cpu().numpy()
    want = oracle.linear(ow, x, fast=True).astype(np.float64)
    assert np.isfinite(got).all()
    for r in range(min(m, 3)):
        f = 1e30 if r == 0 else 1.0
        assert helpers.rel_err(got[r] * f, want[r] * f) < 1e-3


def attention_64(q, kc, vc, start):
    """Causal attention of rows at start .. in 64 bits, and the caches as the kernel reads them: q [s, heads, d]."""
    s, nh, _ = q.shape
    n, rep = start + s, nh // kc.shape[0]
    k, v = (t[:, :n].double().numpy().repeat(rep, 0) for t in (kc, vc))
    sc = np.einsum("shd,hkd->hsk", q.astype(np.float64), k) / np.sqrt(q.shape[2])
    sc[:, np.arange(n)[None] > start + np.arange(s)[:, None]] = -np.inf
    p = np.exp(sc - sc.max(-1, keepdims=True))
    return np.einsum("hsk,hkd->shd", p / p.sum(-1, keepdims=True), v).reshape(s, -1)


def attention_inputs(kind, s, nh, nkv, d, n):
    rng = np.random.default_rng(s + n)
    q, k, v = (rng.normal(size=shape).astype(np.float32) for shape in ((s, nh, d), (nkv, n, d), (nkv, n, d)))
    if kind == "small queries":      # products of ordinary size out of queries that are small in their own type
        q, k = q * 1e-3, k * 1e3
    elif kind == "one-sided values":  # sums that only grow: roundings toward zero add up
        v += 2
    elif kind == "long tail":        # one key far ahead of many whose weights are 1e-6 of its own
        q[:], k, v = 1.0, k * 0.01, v * 0.01 + 1
        k[:, 0] += 14.0 / np.sqrt(d)
        v[:, 0] = -1
    elif kind == "large queries":    # beyond the range of f16
        q, k = q * 1e6, k * 1e-6
    return q, k, v


def rel_64(got, want):
    return np.linalg.norm(got - want) / np.linalg.norm(want)


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("kind", ["normal", "small queries", "large queries", "one-sided values", "long tail"])
@pytest.mark.parametrize("s,start,d", [(1, 4095, 128), (1, 300, 64), (3, 4000, 64), (20, 1000, 128)])
def test_attention_decode_keeps_f32_accuracy(native_lib, dtype, kind, s, start, d):
    """Few rows on 2-byte caches (queries and weights as sums of two or three terms of the cache's type) against 64 bits:
    the terms hold 2^-24 of a query or weight, a step of 16 keys adds at most a handful of truncations of 2^-25, and the
    steps are added up with roundings of 2^-25 either way, which for one-sided sums of 300 steps stays under 2^-20."""
    from dyninfer_b200 import ops
    q, k, v = attention_inputs(kind, s, 8, 2, d, start + s)
    tt = {"bf16": torch.bfloat16, "f16": torch.float16}[dtype]
    kt, vt = torch.from_numpy(k).to(tt), torch.from_numpy(v).to(tt)
    got = ops.attention(torch.from_numpy(q).cuda(), kt.cuda(), vt.cuda(), start).cpu().numpy()
    assert rel_64(got, attention_64(q, kt, vt, start)) < 2.0 ** -20


@pytest.mark.parametrize("kind", ["normal", "small queries", "large queries", "one-sided values", "long tail"])
@pytest.mark.parametrize("s,start,nh,nkv", [(64, 0, 8, 2), (45, 4000, 4, 1), (200, 500, 8, 4)])
def test_attention_prefill_f32_cache_keeps_f32_accuracy(native_lib, kind, s, start, nh, nkv):
    """f16 pairs against 64 bits: a pair holds 2^-24 of a value, scores take chains of four mma, the steps of 32 keys are
    added up with roundings; the bound is the decode kernel's. Equal small addends on a large sum round the same way each
    time: a long tail adds 2^-24 for each of a half's (start + s) / 64 steps, in the sum and in the output."""
    from dyninfer_b200 import ops
    q, k, v = attention_inputs(kind, s, nh, nkv, 128, (start + s + 63) // 64 * 64)
    kt, vt = torch.from_numpy(k), torch.from_numpy(v)
    got = ops.attention(torch.from_numpy(q).cuda(), kt.cuda(), vt.cuda(), start).cpu().numpy()
    bound = 2.0 ** -20 + ((start + s) / 64 * 2.0 ** -23 if kind == "long tail" else 0)
    assert rel_64(got, attention_64(q, kt, vt, start)) < bound


@pytest.mark.parametrize("plane", ["keys", "values"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_attention_prefill_f32_cache_entries_that_are_not_finite(native_lib, plane, bad):
    """A key or value that is not finite reaches the rows that see it and no earlier one, also of the same tile; values far
    beyond f16 beside it keep their accuracy."""
    from dyninfer_b200 import ops
    s, start, at = 100, 20, 70              # row 50 of the chunk writes key 70, in the middle of the second tile
    q, k, v = attention_inputs("normal", s, 4, 2, 128, 128)
    k[:, 64:128] *= 1e3
    v[:, 64:128] *= 1e6
    want = attention_64(q, torch.from_numpy(k), torch.from_numpy(v), start)
    (k if plane == "keys" else v)[1, at, 5] = bad
    got = ops.attention(*(torch.from_numpy(t).cuda() for t in (q, k, v)), start).cpu().numpy().reshape(s, 4, 128)
    want = want.reshape(s, 4, 128)
    assert rel_64(got[:, :2], want[:, :2]) < 2.0 ** -20          # the other kv head
    assert rel_64(got[:at - start], want[:at - start]) < 2.0 ** -20
    assert not np.isfinite(got[at - start:, 2:, 5]).any()


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("s,start,nkv,lost", [(100, 20, 2, [(70, 5)]), (128, 0, 2, [(0, 64), (127, 127)]), (33, 0, 1, [(32, 0), (1, 3)]),
                                              (300, 20, 2, [(31, 5), (32, 5), (190, 77), (319, 0)]), (128, 64, 80, [(65, 1), (130, 2), (191, 126)])])
def test_attention_prefill_2_byte_cache_values_that_are_not_finite(native_lib, dtype, bad, s, start, nkv, lost):
    """A value that is not finite reaches its dim of the rows that see its key, and nothing else: not the earlier rows of
    the same block or tile, not the other dims. First and last keys of tiles and blocks, several in a tile, one and more blocks
    per head; the keys behind the last row are not finite either. Bounds as at the edges of blocks below."""
    from dyninfer_b200 import ops
    d, cap, nh = 128, 1408, 2 * nkv
    g = torch.Generator("cuda").manual_seed(s + start)
    tt = torch.bfloat16 if dtype == "bf16" else torch.float16
    q, k, v = (torch.randn(*shape, generator=g, device="cuda") for shape in ((s, nh, d), (nkv, cap, d), (nkv, cap, d)))
    k, v = k.to(tt), v.to(tt)
    n = start + s
    scores = torch.einsum("shd,hkd->hsk", q.double(), k[:, :n].double().repeat_interleave(2, 0)) / d ** 0.5
    hidden = torch.arange(n, device="cuda")[None, :] > torch.arange(s, device="cuda")[:, None] + start
    want = scores.masked_fill(hidden, float("-inf")).softmax(-1) @ v[:, :n].double().repeat_interleave(2, 0)     # [nh, s, d]
    touched = torch.zeros(nh, s, d, dtype=torch.bool, device="cuda")
    largest = float(v[:, :n].abs().max())
    v[:, n:] = bad
    for key, dim in lost:
        v[0, key, dim] = bad
        touched[:2, max(0, key - start):, dim] = True
    got = ops.attention(q, k, v, start).reshape(s, nh, d).double().transpose(0, 1)
    assert torch.equal(~got.isfinite(), touched)
    assert float((got - want)[~touched].abs().max()) < (1e-4 if dtype == "bf16" else 4e-6) * largest


@pytest.mark.parametrize("hidden,inter", [(2048, 4608), (1024, 4608)])
def test_few_row_steps_where_only_the_fused_matrix_is_large(native_lib, oracle, tmp_path, hidden, inter):
    """gate and up pass for the few-row GEMM one by one, [gate; up] as one matrix does not: prompts and batched steps of 17
    and more rows take another path, as steps of a larger model do."""
    from dyninfer_b200 import checkpoint as ck
    from test_gpu_model import oracle_run
    cfg = dict(synth.SMALL_D128, layers=1, hidden=hidden, intermediate=inter, vocab=512)
    path = synth.write_qwen3_gguf(str(tmp_path / "q.gguf"), cfg, seed=11)
    cat = ck.open_catalog(path)
    prompt = np.random.default_rng(1).integers(0, 512, size=40).tolist()
    want, toks, _ = oracle_run(oracle, cat, prompt, 1, kv_round=2, kv_cap=64)
    model = ModelLoader().load(path, max_kv=64, kv_dtype="bf16", chunk_size=64)
    slots = 18
    with model.create_batched_session(SessionConfig(max_sequence_length=64, batch_size=slots)) as s:
        for b in range(slots):
            lg, _ = s.prefill_slot(b, prompt, want_logits=True)
            assert np.abs(lg - want[0]).max() <= 1e-2
        _, logits = s.step({b: toks[0] for b in range(slots)}, want_logits=True)
        for b in range(slots):
            assert np.abs(logits[b] - want[1]).max() <= 1e-2 and helpers.cosine(logits[b], want[1]) >= 0.9999


@pytest.mark.parametrize("enc", ["gguf.q4_0", "gguf.q8_0", "gguf.q6_k", "gguf.q4_k", "mlx.affine.u4"])
@pytest.mark.parametrize("m,n,k", [(1, 5120, 13824), (1, 4096, 4608), (1, 640, 16384), (1, 1288, 12800), (3, 2560, 2560),
                                   (4, 5120, 5120), (2, 700, 1536)])
def test_linear_few_rows_on_both_sides_of_the_plan_rule(native_lib, oracle, enc, m, n, k):
    """Products whose plan leaves a nearly empty round, too few blocks, or copies per row, and their neighbours: whichever
    kernel takes them, f32 rows keep f32 accuracy."""
    from dyninfer_b200 import ops
    from test_gpu_ops import make_pair
    dw, ow = make_pair(oracle, enc, n, k, seed=n + m)
    x = np.random.default_rng(m).normal(size=(m, k)).astype(np.float32)
    got = ops.linear(dw, torch.from_numpy(x).cuda()).cpu().numpy()
    assert helpers.rel_err(got, oracle.linear(ow, x, fast=True)) < 2e-5


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("s,start,nh,nkv", [(32, 0, 4, 2), (127, 0, 2, 1), (128, 64, 2, 2), (129, 127, 4, 1), (40, 200, 8, 2),
                                            (257, 383, 3, 3), (64, 1087, 2, 1), (300, 20, 80, 8)])
def test_attention_prefill_at_the_edges_of_blocks(native_lib, dtype, s, start, nh, nkv):
    """128-row blocks and 64-key tiles that end on, before and behind a boundary; one to four blocks share the keys, some of
    their streams without a tile; more blocks than SMs. Operands are pairs: 22 bits with f16 terms, 16 with bf16 ones, so that
    an output, a mean of values of size one, is off by a few 2^-22 (2^-16) of their largest."""
    from dyninfer_b200 import ops
    d, cap = 128, 1408
    g = torch.Generator("cuda").manual_seed(s + start)
    q, k, v = (torch.randn(*shape, generator=g, device="cuda") for shape in ((s, nh, d), (nkv, cap, d), (nkv, cap, d)))
    tt = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dtype]
    k, v = k.to(tt), v.to(tt)
    k[:, start + s:] = float("nan")                  # never-written rows must not leak into the result
    v[:, start + s:] = float("inf")
    got = ops.attention(q, k, v, start).reshape(s, nh, d).double()
    hidden = torch.arange(start + s, device="cuda")[None, :] > torch.arange(s, device="cuda")[:, None] + start
    for h in range(nh):
        kh, vh = (c[h // (nh // nkv), :start + s].double() for c in (k, v))
        want = (q[:, h].double() @ kh.T / d ** 0.5).masked_fill(hidden, float("-inf")).softmax(-1) @ vh
        assert float((got[:, h] - want).abs().max()) < (1e-4 if dtype == "bf16" else 4e-6) * float(vh.abs().max())


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("s,start,nh,nkv", [(64, 0, 2, 1), (65, 0, 2, 1), (128, 5, 4, 2), (300, 0, 2, 1), (260, 130, 6, 3), (100, 60, 40, 8)])
def test_attention_prefill_of_few_tiles(native_lib, dtype, s, start, nh, nkv):
    """One to seven tiles: two or four blocks share them, some of which have none, in the last row block or in the first one only."""
    test_attention_prefill_at_the_edges_of_blocks(native_lib, dtype, s, start, nh, nkv)


@pytest.mark.parametrize("enc", ["gguf.q4_0", "gguf.q4_1", "gguf.q8_0", "gguf.q4_k", "mlx.affine.u4"])
@pytest.mark.parametrize("m,n,k", [(33, 130, 256), (48, 127, 768), (49, 1000, 2560), (64, 257, 3072), (47, 2049, 1792),
                                   (64, 6000, 1024), (40, 128, 6144), (64, 129, 6400), (65, 1024, 2048), (128, 257, 1536),
                                   (100, 2048, 2048), (127, 1000, 3072)])
def test_linear_rows_over_a_cluster(native_lib, oracle, enc, m, n, k):
    """33 to 128 rows, K over clusters of two to eight blocks with one to three units each (and sizes beyond): ragged
    tiles and row groups, a last block with fewer units, odd row counts per finishing block. Both operands are rounded to
    2^-12 of a value; over k products the error of a sum, relative to its size, is about 2^-12 * sqrt(2 / 3) = 2.0e-4 (rounding
    errors are uniform), so 4e-4 over all outputs holds with room."""
    from dyninfer_b200 import ops
    from test_gpu_ops import make_pair
    if enc == "mlx.affine.u4" and k % 512:
        pytest.skip("the few-row kernels take MLX rows of whole 512s")
    dw, ow = make_pair(oracle, enc, n, k, seed=n + m)
    x = np.random.default_rng(m).normal(size=(m, k)).astype(np.float32)
    got = ops.linear(dw, torch.from_numpy(x).cuda()).cpu().numpy()
    assert helpers.rel_err(got, oracle.linear(ow, x, fast=True)) < 4e-4


# encoding, activation rows, matrix rows, K, MLX group and type of scales; that the GEMM over a cluster takes them: test_gemm_cluster_plan.py
CLUSTER_PRODUCTS = [("gguf.q5_k", 65, 1000, 2048, 0, ""), ("gguf.q5_k", 128, 257, 1536, 0, ""), ("gguf.q5_k", 99, 2048, 2560, 0, ""),
                    ("mlx.affine.u4", 48, 1000, 2048, 32, "bf16"), ("mlx.affine.u4", 64, 257, 1024, 32, "f16"),
                    ("mlx.affine.u4", 65, 1000, 1792, 32, "f32"), ("mlx.affine.u4", 128, 300, 2304, 64, "bf16"),
                    ("mlx.affine.u4", 100, 2048, 2048, 128, "f32"), ("mlx.affine.u4", 66, 129, 2816, 256, "f16")]


@pytest.mark.parametrize("enc,m,n,k,group,aux", CLUSTER_PRODUCTS)
def test_linear_encodings_over_a_cluster(native_lib, oracle, enc, m, n, k, group, aux):
    """Q5_K (65 rows and more only), MLX groups of 32 to 256, scales of every type and rows of an odd multiple of 256. The bound is that of
    test_linear_rows_over_a_cluster."""
    from dyninfer_b200 import ops
    t = synth.random_weight(enc, n, k, m + n, **({"group": group} if group else {}))
    if group:
        scales, biases = (synth.bf16_bits_to_f32(t[c]) for c in ("scales", "biases"))
        if aux == "f16":
            scales, biases = scales.astype(np.float16), biases.astype(np.float16)
        if aux == "bf16":
            scales, biases = t["scales"], t["biases"]
        args = (enc, n, k, t["packed"], scales, biases, "plain." + aux, group)
    else:
        args = (enc, n, k, t["data"])
    x = np.random.default_rng(m).normal(size=(m, k)).astype(np.float32)
    got = ops.linear(ops.DeviceWeight(*args), torch.from_numpy(x).cuda()).cpu().numpy()
    assert helpers.rel_err(got, oracle.linear(oracle.Weight(*args), x, fast=True)) < 4e-4


def test_linear_over_a_cluster_on_two_streams(native_lib, oracle):
    """Products of plans with 256 and with 512 columns of tensor memory, on two streams at a time (blocks of both kinds are kept off
    one SM: test_gemm_cluster_plan.py). Each gives the bits that it gives alone."""
    from dyninfer_b200 import ops
    from test_gpu_ops import make_pair
    ws = [make_pair(oracle, "gguf.q4_0", n, 1024, seed=n)[0] for n in (4096, 6144, 1024)]
    xs = [torch.randn(m, 1024, generator=torch.Generator("cuda").manual_seed(m), device="cuda") for m in (64, 40)]
    want = [[ops.linear(w, x) for w in ws] for x in xs]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in xs], [[], []]
    for i in range(30):
        for j, (stream, x) in enumerate(zip(streams, xs)):
            with torch.cuda.stream(stream):
                got[j].append(ops.linear(ws[(i + j) % 3], x))
    torch.cuda.synchronize()
    ops.check_device_error()
    for j in range(2):
        assert all(torch.equal(y, want[j][(i + j) % 3]) for i, y in enumerate(got[j]))


@pytest.mark.parametrize("hidden", [1280, 1536, 2816, 3584, 7168, 1344])
def test_many_row_norm_widths(native_lib, oracle, tmp_path, hidden):
    """Rows that are multiples of 256 but not of 1024 elements (the last runs of a thread stay empty), and one that is
    neither: 80 rows through layers whose norms write the GEMM's operand, K-split sums added in front of them. (Typical
    difference 3e-4 to 1e-3. A random prompt can end on a token that amplifies roundings: with seed 2 at 1536 the oracle's
    own two summation orders are 1e-3 apart and every version of the f16 path 1.5e-2.)"""
    from dyninfer_b200 import checkpoint as ck
    from test_gpu_model import oracle_run
    cfg = dict(synth.SMALL_D128, hidden=hidden, intermediate=512, vocab=512)
    path = synth.write_qwen3_gguf(str(tmp_path / "q.gguf"), cfg, seed=13, embd="gguf.q8_0")
    cat = ck.open_catalog(path)
    prompt = np.random.default_rng(3).integers(0, 512, size=80).tolist()
    want, _, _ = oracle_run(oracle, cat, prompt, 0, kv_round=2, kv_cap=128)
    model = ModelLoader().load(path, max_kv=128, kv_dtype="bf16", chunk_size=128)
    with model.create_session(SessionConfig(max_sequence_length=128)) as s:
        got = s.prefill(prompt).values
    assert np.abs(got - want[0]).max() <= 1e-2 and helpers.cosine(got, want[0]) >= 0.9999


@pytest.mark.parametrize("enc", ["gguf.q4_0", "gguf.q8_0", "gguf.q4_k", "mlx.affine.u4"])
@pytest.mark.parametrize("m,n,k", [(256, 4096, 8192), (300, 1024, 8192), (300, 640, 8192), (160, 3500, 8192),
                                   (1100, 3500, 8192), (1100, 3500, 12288), (2048, 2300, 12288)])
def test_linear_many_rows_where_a_k_split_fills_the_gpu(native_lib, oracle, enc, m, n, k):
    """A long K split over about as many blocks as there are SMs, and its neighbours that are cut into equal shares."""
    from dyninfer_b200 import ops
    from test_gpu_ops import make_pair
    dw, ow = make_pair(oracle, enc, n, k, seed=n + m)
    x = np.random.default_rng(m).normal(size=(m, k)).astype(np.float32)
    rows = [0, 63, 127, 128, m - 1]
    got = ops.linear(dw, torch.from_numpy(x).cuda()).cpu().numpy()
    want = oracle.linear(ow, x[rows], fast=True)
    assert helpers.rel_err(got[rows], want) < 1e-3


@pytest.mark.parametrize("enc", ["plain.bf16", "plain.f16"])
@pytest.mark.parametrize("m,n,k", [(5, 4096, 4096), (8, 3072, 1024), (9, 520, 2560), (16, 4096, 4096)])
def test_linear_few_rows_of_plain_weights_keep_f32_accuracy(native_lib, enc, m, n, k):
    """5 to 16 f32 rows against 64 bits: the terms hold 2^-24 of a value, a unit of K adds chains of up to eight mma at 2^-26
    of the sum each, the units are added with roundings of 2^-25."""
    from dyninfer_b200 import ops
    w = ops.DeviceWeight(enc, n, k, synth.random_weight(enc, n, k, seed=m)["data"])
    x = torch.randn(m, k, generator=torch.Generator("cuda").manual_seed(m), device="cuda")
    want = (x.double() @ ops.dequant(w).double().T).cpu().numpy()
    assert rel_64(ops.linear(w, x).double().cpu().numpy(), want) < 2.0 ** -21


EDGES = [0, 1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 299]


def one_by_one(oracle, path, tokens, at, kv):
    """The oracle's logits after each of the positions in `at`, the cache rounded to its type."""
    from dyninfer_b200 import checkpoint as ck
    cat = ck.open_catalog(path)
    m = oracle.Model(cat.config, helpers.catalog_weights(oracle, cat), kv_cap=len(tokens), kv_round={"f16": 1, "bf16": 2, "f32": 0}[kv], fast=True)
    out = {}
    for i, t in enumerate(tokens):
        lg, _ = m.forward([t])
        if i in at:
            out[i] = lg
    return out


@pytest.mark.parametrize("kv", ["bf16", "f16"])
@pytest.mark.parametrize("d,slots", [(128, 1), (64, 1), (128, 3)])
def test_decode_attention_prepares_its_own_rows(native_lib, oracle, tmp_path, kv, d, slots):
    """Decode attention with the QKV preparation inside (norm, rotation, cache write, the slice that owns the new key) at
    every position around the ends of its slices, token by token against the oracle. The products in front keep 22 bits of
    their rows and the attention 24, so what is left are roundings of single cache entries that fall the other way:
    2^-9 (bf16) or 2^-12 of an entry."""
    cfg = dict(synth.TINY, layers=1, heads=8, kv_heads=2, head_dim=d, hidden=512)
    path = synth.write_qwen3_gguf(str(tmp_path / "q.gguf"), cfg, seed=17)
    rng = np.random.default_rng(d + slots)
    tokens = [rng.integers(0, cfg["vocab"], size=max(EDGES) + 1).tolist() for _ in range(slots)]
    want = [one_by_one(oracle, path, t, EDGES, kv) for t in tokens]
    model = ModelLoader().load(path, max_kv=512, kv_dtype=kv, chunk_size=1, decode_kernel="graph")
    if slots == 1:
        with model.create_session(SessionConfig(max_sequence_length=512)) as s:
            for i, t in enumerate(tokens[0]):
                lg = (s.prefill([t]) if i == 0 else s.decode(t)).values
                if i in want[0]:
                    assert np.abs(lg - want[0][i]).max() <= 1e-3, i
        return
    with model.create_batched_session(SessionConfig(max_sequence_length=512, batch_size=slots)) as s:
        for b in range(slots):
            s.prefill_slot(b, tokens[b][:1])
        for i in range(1, len(tokens[0])):
            _, logits = s.step({b: tokens[b][i] for b in range(slots)}, want_logits=True)
            if i in want[0]:
                for b in range(slots):
                    assert np.abs(logits[b] - want[b][i]).max() <= 1e-3, (i, b)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("rows", [127, 128, 296, 297, 593])
def test_prompt_rows_prepared_by_fewer_blocks(native_lib, oracle, tmp_path, rows, d):
    """Prompts of one chunk whose rows are prepared for the attention by a block per eight heads, two blocks, one block, and
    more blocks than fit at once; 20 heads, so the last warps of a block have fewer. f16 operands of the products: 1e-2."""
    cfg = dict(synth.TINY, layers=1, heads=12, kv_heads=4, head_dim=d, hidden=512)
    path = synth.write_qwen3_gguf(str(tmp_path / "q.gguf"), cfg, seed=23)
    prompt = np.random.default_rng(rows).integers(0, cfg["vocab"], size=rows).tolist()
    want = one_by_one(oracle, path, prompt, [rows - 1], "bf16")[rows - 1]
    model = ModelLoader().load(path, max_kv=1024, kv_dtype="bf16", chunk_size=1024)
    with model.create_session(SessionConfig(max_sequence_length=1024)) as s:
        got = s.prefill(prompt).values
    assert np.abs(got - want).max() <= 1e-2 and helpers.cosine(got, want) >= 0.9999


@pytest.mark.parametrize("kv", ["bf16", "f16"])
@pytest.mark.parametrize("slots", [8, 40])
def test_batched_decode_attention_at_the_ends_of_slices(native_lib, oracle, tmp_path, kv, slots):
    """Steps of many sequences (slices that meet in a cluster, and more blocks than SMs: slices through memory) whose
    contexts end around the ends of the slices, against the oracle; f16 operands of the products in front: 1e-2."""
    cfg = dict(synth.SMALL_D128, layers=1, heads=8, kv_heads=4, vocab=512)
    path = synth.write_qwen3_gguf(str(tmp_path / "q.gguf"), cfg, seed=19)
    rng = np.random.default_rng(slots)
    lengths = [EDGES[1:][(5 * b) % (len(EDGES) - 1)] for b in range(slots)]
    tokens = [rng.integers(0, 512, size=n + 1).tolist() for n in lengths]
    model = ModelLoader().load(path, max_kv=320, kv_dtype=kv, chunk_size=64, decode_kernel="graph")
    with model.create_batched_session(SessionConfig(max_sequence_length=320, batch_size=slots)) as s:
        for b in range(slots):
            s.prefill_slot(b, tokens[b][:-1])
        _, logits = s.step({b: tokens[b][-1] for b in range(slots)}, want_logits=True)
    for b in range(slots):
        want = one_by_one(oracle, path, tokens[b], [lengths[b]], kv)[lengths[b]]
        assert np.abs(logits[b] - want).max() <= 1e-2 and helpers.cosine(logits[b], want) >= 0.9999, (b, lengths[b])


def test_persistent_attention_slices_against_the_oracle(native_lib, oracle, tmp_path):
    """One slice of a head's keys up to the most there are (nine, then several batches per slice), token by token."""
    path = synth.write_qwen3_gguf(str(tmp_path / "q.gguf"), dict(synth.SMALL_D128, vocab=512), seed=5)
    at = [0, 62, 63, 64, 127, 128, 191, 192, 511, 512, 575, 576, 577, 1030]
    tokens = np.random.default_rng(3).integers(0, 512, size=max(at) + 1).tolist()
    want = one_by_one(oracle, path, tokens, at, "bf16")
    model = ModelLoader().load(path, max_kv=1152, kv_dtype="bf16", chunk_size=128, decode_kernel="persistent")
    with model.create_session(SessionConfig(max_sequence_length=1152)) as s:
        assert s.uses_persistent_kernel()
        for i, t in enumerate(tokens):
            lg = (s.prefill([t]) if i == 0 else s.decode(t)).values
            if i in want:
                assert np.abs(lg - want[i]).max() <= 1e-2 and helpers.cosine(lg, want[i]) >= 0.9999, i


@pytest.mark.parametrize("hidden,inter,group", [(1024, 1536, 64), (1024, 1536, 32), (1024, 1536, 128), (1536, 2304, 64),
                                                (512, 768, 32), (512, 4096, 64), (2048, 256, 128)])
def test_persistent_mlx_widths_and_groups(native_lib, tmp_path, hidden, inter, group):
    """One slice of K and several, shares of two to sixteen blocks per warp, every group size, gate and up rows in one tile: the
    persistent kernel against the operator path (both keep f32 rows to 22 bits)."""
    cfg = dict(synth.SMALL_D64, hidden=hidden, intermediate=inter, vocab=512)
    path = synth.write_qwen3_mlx(str(tmp_path / "mlx"), cfg, seed=9, group=group)
    got = []
    for kernel in ("persistent", "graph"):
        model = ModelLoader().load(path, max_kv=64, kv_dtype="f32", chunk_size=64, decode_kernel=kernel)
        with model.create_session(SessionConfig(max_sequence_length=64)) as s:
            assert s.uses_persistent_kernel() == (kernel == "persistent")
            s.prefill([3])
            got.append(np.stack([s.decode(t).values.copy() for t in (7, 11, 400)]))
    assert np.abs(got[0] - got[1]).max() <= 1e-4 * np.abs(got[1]).max()


@pytest.mark.parametrize("hidden,inter,group", [(2048, 4096, 128), (1536, 4608, 64), (1536, 6144, 32), (512, 1536, 64)])
def test_persistent_mlx_gate_and_up_by_tiles(native_lib, tmp_path, hidden, inter, group):
    """As many tiles on the busiest block with gate and up in one as with each in its own: apart for several slices of K, together for one."""
    test_persistent_mlx_widths_and_groups(native_lib, tmp_path, hidden, inter, group)


@pytest.mark.parametrize("enc", ["gguf.q4_0", "gguf.q8_0"])
@pytest.mark.parametrize("kv", ["bf16", "f16", "f32"])
def test_few_row_chains_give_the_same_bits_every_time(native_lib, tmp_path, enc, kv):
    """Many small layers as one chain of dependent launches: prompts and batched steps of every kind of row count, repeated
    on a session whose buffers hold other values from prompt to prompt, are finite and do not change by a bit."""
    cfg = dict(synth.SMALL_D128, layers=16, heads=8, kv_heads=4, intermediate=3072, vocab=512)
    path = synth.write_qwen3_gguf(str(tmp_path / "q.gguf"), cfg, seed=23, encodings=dict.fromkeys(synth.linear_shapes(cfg), enc),
                                  repeat_layers=True)
    rng = np.random.default_rng(7)
    model = ModelLoader().load(path, max_kv=256, kv_dtype=kv, chunk_size=64)
    prompts = {n: rng.integers(0, 512, size=n).tolist() for n in (2, 4, 5, 9, 16, 17, 20, 24, 28, 31, 32, 48, 64, 92)}
    first = {}
    with model.create_session(SessionConfig(max_sequence_length=256)) as s:
        for _ in range(6):
            for n, p in prompts.items():
                got = s.prefill(p).values
                assert np.isfinite(got).all(), n
                assert np.array_equal(got, first.setdefault(n, got)), n
    for slots in (3, 8, 24, 40):
        with model.create_batched_session(SessionConfig(max_sequence_length=256, batch_size=slots)) as s:
            seen = None
            for _ in range(4):
                for b in range(slots):
                    s.prefill_slot(b, prompts[28])
                _, logits = s.step({b: 5 + b for b in range(slots)}, want_logits=True)
                logits = np.array([logits[b] for b in range(slots)])
                assert np.isfinite(logits).all()
                seen = logits if seen is None else seen
                assert np.array_equal(logits, seen), slots
