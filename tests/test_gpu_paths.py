"""Kernel variants at the sizes where their dispatch or their tiling changes, against the CPU oracle."""
import numpy as np
import pytest

import helpers

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
