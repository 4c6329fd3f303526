"""The builder's passes over the elements where their form changes, byte for byte against the oracle: pieces of eight and of
four elements, segments whose counters a warp walks and a CTA shares, items sorted by one, two and three bytes of their
counts, and codes put side by side in fours and pairs with ESC codes among them."""
import numpy as np
import pytest
import torch

import MPServe_cuda
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _same(built, want):
    assert set(built) == set(want)
    for key, ref in want.items():
        mine = built[key].cpu()
        mine = mine.view(torch.uint16).numpy() if mine.dtype == torch.bfloat16 else mine.numpy()
        np.testing.assert_array_equal(mine, ref, err_msg=key)


def _on_device(sym, ctx, shift):
    """The two arrays `shift` elements behind the start of an allocation."""
    def put(a):
        buf = torch.zeros(a.size + 16, dtype=torch.uint8 if a.dtype == np.uint8 else torch.uint16, device="cuda")
        view = buf[shift:shift + a.size].view(a.shape)
        view.copy_(torch.from_numpy(a))
        return view
    return put(sym).view(torch.bfloat16), put(ctx)


@pytest.mark.parametrize("n,m,shift,k", [(40, 1024, 0, 64), (40, 1024, 8, 64), (40, 1024, 4, 64), (41, 1020, 0, 60), (40, 1024, 1, 64),
                                         (17, 8200, 0, 1024), (3000, 8, 0, 256)])
def test_pieces(n, m, shift, k):
    rng = np.random.default_rng(n + m + shift)
    ctx = rng.integers(0, 256, (n, m)).astype(np.uint8)
    sym = (0x3000 + (ctx.astype(np.int64) & 0x7F) * 8 + rng.integers(0, 20, (n, m)) + ((ctx.astype(np.int64) >> 7) << 15)).astype(np.uint16)
    sc = (0x3F00 + np.arange(n) % 2).astype(np.uint16)
    w, c = _on_device(sym, ctx, shift)
    built = MPServe_cuda.huffman_build_fp8_decode_tables(w, c, torch.from_numpy(sc).cuda(), max_len=7, threads_per_block=k)
    _same(built, orc.build_fp8(sym, ctx, sc, 7, k))


@pytest.mark.parametrize("positive,negative", [(1022, 1), (1023, 0), (1024, 0), (0, 1024), (1024, 1), (500, 524), (40, 3000), (3000, 40),
                                               (2047, 2049), (8192, 8192)])
def test_wide_contexts(positive, negative):
    """Context 3 sees every `step`-th symbol of a range of either sign; the counters are as many as the ranges are wide."""
    rng = np.random.default_rng(positive * 7 + negative)
    values = np.concatenate([np.arange(0, positive, 3), [positive - 1] if positive else [], 0x8000 + np.arange(0, negative, 5),
                             [0x8000 + negative - 1] if negative else []]).astype(np.int64)
    n, m = 64, 1024
    sym = rng.choice(values, n * m)
    sym[:values.size] = values
    ctx = np.full(n * m, 3)
    other = rng.random(n * m) < 0.3
    other[:values.size] = False
    sym = np.where(other, 0x3C00 + rng.integers(0, 9, n * m), sym)
    ctx = np.where(other, 4 + rng.integers(0, 4, n * m), ctx)
    order = rng.permutation(n * m)
    sym, ctx = sym[order].astype(np.uint16).reshape(n, m), ctx[order].astype(np.uint8).reshape(n, m)
    sc = np.array([77], dtype=np.uint16)
    w = torch.from_numpy(sym).view(torch.bfloat16).cuda(), torch.from_numpy(ctx).cuda(), torch.from_numpy(sc).cuda()
    _same(MPServe_cuda.huffman_build_fp8_decode_tables(*w, max_len=7, threads_per_block=128), orc.build_fp8(sym, ctx, sc, 7, 128))
    _same(MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables_by_scale(*w, max_len=11, threads=128, group_cap=9),
          orc.build_awq_by_scale(sym, ctx, sc, 11, 128, 9))


@pytest.mark.parametrize("L", [7, 8, 9, 11, 12])
@pytest.mark.parametrize("distinct,most", [(33, 255), (33, 256), (100, 300), (128, 70000), (300, 255), (300, 66000), (513, 300), (700, 257)])
def test_sorted_by_count(distinct, most, L):
    """One context; many symbols of equal count, one that occurs `most` times."""
    rng = np.random.default_rng(distinct + most + L)
    counts = rng.integers(1, 6, distinct) + 255 * (rng.random(distinct) < 0.05)
    counts[rng.integers(distinct)] = most
    sym = np.repeat(rng.choice(65536, distinct, replace=False), counts)
    sym = np.concatenate([sym, np.repeat(sym[:1], -sym.size % 64)])
    rng.shuffle(sym)
    sym = sym.astype(np.uint16).reshape(-1, 64)
    ctx = np.zeros(sym.shape, np.uint8)
    sc = np.array([5], dtype=np.uint16)
    w = torch.from_numpy(sym).view(torch.bfloat16).cuda(), torch.from_numpy(ctx).cuda(), torch.from_numpy(sc).cuda()
    _same(MPServe_cuda.huffman_build_fp8_decode_tables(*w, max_len=L, threads_per_block=100), orc.build_fp8(sym, ctx, sc, L, 100))
    _same(MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables(*w, max_len=L, threads_per_block=64),
          orc.build_awq_bucket(sym, ctx, sc, L, 64))


@pytest.mark.parametrize("L,k,n,m", [(7, 256, 130, 1024), (8, 512, 130, 1024), (9, 256, 70, 1016), (11, 64, 70, 1024), (12, 256, 130, 1000),
                                     (7, 1000, 100, 3000), (8, 1024, 129, 2053)])
def test_codes_in_groups(L, k, n, m):
    """Contexts of more symbols than table slots beside small ones: groups with and without ESC codes, sub-streams that end
    inside a group."""
    rng = np.random.default_rng(L * k + m)
    ctx = rng.integers(0, 8, (n, m)).astype(np.uint8)
    sym = np.where(ctx == 0, rng.zipf(1.3, (n, m)) % (3 << L), 0x3C00 + rng.integers(0, 12, (n, m))).astype(np.uint16)
    sc = np.array([9], dtype=np.uint16)
    w = torch.from_numpy(sym).view(torch.bfloat16).cuda(), torch.from_numpy(ctx).cuda(), torch.from_numpy(sc).cuda()
    _same(MPServe_cuda.huffman_build_fp8_decode_tables(*w, max_len=L, threads_per_block=k), orc.build_fp8(sym, ctx, sc, L, k))


@pytest.mark.parametrize("scales,m", [(256, 8192), (257, 8192), (3, 8196)])
def test_segments_of_many_scales(scales, m):
    """As many segments as one launch sums up and a scale more; rows that are the bucket lists' and rows cut into pieces."""
    rng = np.random.default_rng(scales)
    n = max(scales, 4)
    ctx = rng.integers(0, 5, (n, m)).astype(np.uint8)
    sym = (0x3000 + ctx.astype(np.int64) * 64 + rng.integers(0, 7, (n, m))).astype(np.uint16)
    sc = (0x2000 + 3 * rng.permutation(np.arange(n) % scales)).astype(np.uint16)
    w = torch.from_numpy(sym).view(torch.bfloat16).cuda(), torch.from_numpy(ctx).cuda(), torch.from_numpy(sc).cuda()
    _same(MPServe_cuda.huffman_build_fp8_decode_tables(*w, max_len=7, threads_per_block=1024), orc.build_fp8(sym, ctx, sc, 7, 1024))
