"""Kernels of the wide decode step at the edges of their splits: the narrow int4 GEMM (one to sixteen rows, dealt to
the warps of one CTA as runs of tiles) and the streaming attention (rounds of 16 or 32 keys over key splits)."""
import numpy as np
import pytest

from test_gpu_ops import bf16_round, make_matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [1, 8, 9, 16])
@pytest.mark.parametrize("n,k,ksplit", [
    (16, 64, 1),            # one tile: fifteen idle warps
    (1152, 1088, 1),        # 17 k tiles
    (2560, 640, 5),         # two k tiles a split
    (40000, 192, 1),        # more row tiles than CTAs: whole row tiles of a warp beside shared ones
])
def test_narrow_gemm(pkg, orc, mio, t, n, k, ksplit):
    packed, scale = make_matrix(mio, n, k, n + k)
    a = bf16_round(np.random.Generator(np.random.PCG64(t)).standard_normal((t, k), dtype=np.float32))
    want = orc.matmul_w4(packed, scale, a)
    got, _ = pkg.ops.gemm_w4(packed, scale, a, mode=pkg.GEMM_TCGEN05, ksplit=ksplit)
    assert np.abs(got - want).max() / np.abs(want).max() < 2e-5


@pytest.mark.parametrize("t,ffn,k", [(1, 64, 64), (9, 192, 320), (16, 4800, 192), (5, 6912, 1152)])
def test_narrow_geglu(pkg, orc, mio, t, ffn, k):
    gp, gs = make_matrix(mio, ffn, k, 1)
    up, us = make_matrix(mio, ffn, k, 2)
    a = bf16_round(np.random.Generator(np.random.PCG64(3)).standard_normal((t, k), dtype=np.float32))
    g = orc.matmul_w4(gp, gs, a).astype(np.float64)
    u = orc.matmul_w4(up, us, a).astype(np.float64)
    want = 0.5 * g * (1 + np.tanh(0.7978845608028654 * (g + 0.044715 * g ** 3))) * u
    got = pkg.ops.gemm_geglu_w4(gp, gs, up, us, a, mode=pkg.GEMM_TCGEN05)
    assert np.abs(got - want).max() / np.abs(want).max() < 1e-2          # output stored as bf16


@pytest.mark.parametrize("hq,hkv,hd,s,window,kv_bf16,nsplit", [
    (4, 1, 256, 1, 0, False, 2),            # one key, an empty split
    (4, 1, 256, 33, 0, False, 2),           # rounds of 16 keys: 16 + 1 and 16
    (4, 2, 256, 96, 0, True, 3),            # rounds of 32 keys that end with the split
    (2, 2, 64, 400, 130, False, 3),         # a window that starts inside a page, splits that cross pages
    (8, 2, 128, 700, 0, True, 16),
])
def test_streaming_attention_rounds(pkg, orc, hq, hkv, hd, s, window, kv_bf16, nsplit):
    rng = np.random.Generator(np.random.PCG64(s))
    q = rng.standard_normal((3, hq, hd), dtype=np.float32)
    k, v = (rng.standard_normal((s, hkv, hd), dtype=np.float32) for _ in range(2))
    kk, vv = (bf16_round(k), bf16_round(v)) if kv_bf16 else (k, v)
    want = np.concatenate([orc.attention(q[i:i + 1], kk, vv, s - 1, window) for i in range(3)])
    got, _ = pkg.ops.attention(q, k, v, window=window, kv_bf16=kv_bf16, nsplit=nsplit, streaming_kernel=True, private_caches=True)
    assert np.abs(got - want).max() < 1e-5, np.abs(got - want).max()
