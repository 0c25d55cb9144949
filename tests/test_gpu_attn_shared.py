"""Decode attention of many queries over one cache (B200LmOps_AttentionDecodeStatic): every row-tile variant, edges of
the 16-key chunks, pages and windows, one split and many, against fp64 softmax attention."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(q, k, v, table, s, window):
    b, hq, hd = q.shape
    hkv = k.shape[1]
    lo = max(0, s - window) if window > 0 else 0
    kk = k[table.long()].transpose(1, 2).reshape(-1, hkv, hd)[lo:s].double()
    vv = v[table.long()].transpose(1, 2).reshape(-1, hkv, hd)[lo:s].double()
    qq = q.double().reshape(b, hkv, hq // hkv, hd)
    p = torch.softmax(torch.einsum("bkgd,skd->bkgs", qq, kk) / hd ** 0.5, dim=-1)
    return torch.einsum("bkgs,skd->bkgd", p, vv).reshape(b, hq, hd)


@pytest.mark.parametrize("hq,hkv,hd", [(4, 1, 256), (8, 4, 128), (2, 2, 64), (4, 2, 32)])
@pytest.mark.parametrize("batch,s,window", [
    (1, 1, 0), (1, 16, 0), (1, 1000, 0), (1, 5000, 512),       # at most four rows: packed terms
    (3, 17, 0), (4, 777, 100), (7, 300, 0), (8, 2049, 0),      # 5 .. 32 rows
    (9, 257, 0), (33, 1023, 256), (64, 3000, 0),               # row tiles with a remainder; more than one tile
])
@pytest.mark.parametrize("bf16", [False, True])
def test_shared_cache_attention_matches_fp64(pkg, hq, hkv, hd, batch, s, window, bf16, nan_ahead=False):
    gen = torch.Generator(device="cuda").manual_seed(batch * 1000 + s)
    pages = -(-s // 256)
    q = torch.randn(batch, (hq + 2 * hkv) * hd, device="cuda", generator=gen)
    kv = torch.bfloat16 if bf16 else torch.float32
    k = torch.randn(pages, hkv, 256, hd, device="cuda", generator=gen).to(kv)
    v = torch.randn(pages, hkv, 256, hd, device="cuda", generator=gen).to(kv)
    k[-1, :, s - (pages - 1) * 256:] = float("nan")            # slots past the last key are never read
    v[-1, :, s - (pages - 1) * 256:] = float("nan")
    k[-1], v[-1] = k[-1].clone(), v[-1].clone()
    if nan_ahead:                                              # nor do those ahead of a window's first key enter
        for p in range(pages):
            k[p, :, :max(0, s - window - 256 * p)] = float("nan")
            v[p, :, :max(0, s - window - 256 * p)] = float("nan")
    table = torch.randperm(pages, device="cuda", generator=gen).to(torch.int32)
    inv = torch.empty_like(table)
    inv[table.long()] = torch.arange(pages, device="cuda", dtype=torch.int32)
    kp, vp = k[inv.long()].contiguous(), v[inv.long()].contiguous()       # logical page i lies at table[i]
    out = torch.full((batch, hq, hd), float("nan"), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    for _ in range(2):                                         # the second call finds the tickets of the first at zero
        pkg.ops.attention_decode_static(q.data_ptr(), kp.data_ptr(), vp.data_ptr(), table.data_ptr(), out.data_ptr(), batch, s, hq, hkv,
                                        hd, window=window, kv_bf16=bf16, nsplit=1, stream=stream)
    assert pkg.ops.attention_decode_static_status(stream=stream) == 0
    want = reference(q[:, :hq * hd].reshape(batch, hq, hd), kp, vp, table, s, window)
    err = ((out.double() - want).norm() / want.norm()).item()
    assert err < 2e-6, err


@pytest.mark.parametrize("batch,s,window,hq,hkv,hd", [
    (16, 1000, 0, 4, 1, 256), (33, 1023, 1001, 4, 1, 256),      # the shortest, a row tile and four rows, both ends inside a tile
    (64, 4097, 0, 4, 1, 256), (32, 1281, 0, 4, 1, 128),
    (10, 8001, 0, 4, 1, 256), (20, 2500, 0, 8, 4, 128),         # at most 48 rows
    (49, 3000, 1500, 2, 2, 128), (64, 1700, 0, 32, 16, 128),    # a group of one; 16 units
    (64, 1100, 0, 32, 32, 128),                                 # as many units as leave one split each
])
def test_many_rows_on_tcgen05(pkg, batch, s, window, hq, hkv, hd):
    assert pkg.ops.attention_decode_static_clusters(batch, s, hq, hkv, hd, window, True) >= 1
    test_shared_cache_attention_matches_fp64(pkg, hq, hkv, hd, batch, s, window, True)


@pytest.mark.parametrize("batch,s,window,hq,hkv,hd", [
    (33, 1023, 1001, 4, 1, 256), (64, 3000, 1500, 4, 1, 128),   # first keys 22 and 28 of a tile of 32
    (64, 4097, 4096, 4, 1, 256), (49, 2600, 1513, 2, 2, 128),   # the second, and the last of a tile in the middle of a page
])
def test_nothing_ahead_of_a_window_enters_on_tcgen05(pkg, batch, s, window, hq, hkv, hd):
    assert pkg.ops.attention_decode_static_clusters(batch, s, hq, hkv, hd, window, True) >= 1
    test_shared_cache_attention_matches_fp64(pkg, hq, hkv, hd, batch, s, window, True, nan_ahead=True)


@pytest.mark.parametrize("batch,s,window,hq,hkv,hd,bf16,tcgen05", [
    (8, 32768, 0, 4, 1, 256, True, False), (9, 32768, 0, 4, 1, 256, True, True),       # 32 and 36 rows
    (12, 7999, 0, 4, 1, 256, True, False), (12, 8000, 0, 4, 1, 256, True, True),       # 48: keys of all kv heads
    (20, 2499, 0, 8, 4, 128, True, False), (20, 2500, 0, 8, 4, 128, True, True),       # and of one
    (13, 999, 0, 4, 1, 256, True, False), (13, 1000, 0, 4, 1, 256, True, True),        # 52
    (64, 5000, 999, 4, 1, 128, True, False), (64, 5000, 1000, 4, 1, 128, True, True),  # a window's keys are what counts
    (64, 5000, 0, 4, 1, 256, False, False), (64, 5000, 0, 2, 2, 64, True, False),      # other caches and head sizes
])
def test_which_calls_run_on_tcgen05(pkg, batch, s, window, hq, hkv, hd, bf16, tcgen05):
    assert (pkg.ops.attention_decode_static_clusters(batch, s, hq, hkv, hd, window, bf16) > 0) == tcgen05
    test_shared_cache_attention_matches_fp64(pkg, hq, hkv, hd, batch, s, window, bf16)


def test_unaligned_cache_goes_through_the_plain_kernel(pkg):
    gen = torch.Generator(device="cuda").manual_seed(5)
    s, hd = 300, 32
    raw = [torch.randn(2 * 256 * hd + 1, device="cuda", generator=gen)[1:] for _ in range(2)]     # 4 bytes off
    k, v = (r.reshape(2, 1, 256, hd) for r in raw)
    q = torch.randn(3, 4 * hd + 2 * hd, device="cuda", generator=gen)
    table = torch.arange(2, device="cuda", dtype=torch.int32)
    out = torch.empty(3, 4, hd, device="cuda")
    pkg.ops.attention_decode_static(q.data_ptr(), k.data_ptr(), v.data_ptr(), table.data_ptr(), out.data_ptr(), 3, s, 4, 1, hd, nsplit=2,
                                    stream=torch.cuda.current_stream().cuda_stream)
    want = reference(q[:, :4 * hd].reshape(3, 4, hd), k, v, table, s, 0)
    assert ((out.double() - want).norm() / want.norm()).item() < 2e-6
