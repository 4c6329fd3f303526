"""The counting histogram of the sidecar builder against the oracle, where its form changes: scales with enough elements
for it and scales without, ranges of symbols too wide for its counters, values of both signs and zeros of either, rows of
several pieces with a short last one, blocks of rows, and stretches of rows that end inside a scale."""
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


def _weight(n, m, spread, seed):
    """Symbols near a pattern that the context chooses, of either sign, `spread` of them; a few zeros."""
    rng = np.random.default_rng(seed)
    ctx = rng.integers(0, 256, (n, m)).astype(np.uint8)
    sym = (0x3000 + (ctx.astype(np.int64) & 0x7F) * 8 + rng.integers(0, spread, (n, m))) & 0x7FFF
    sym |= (ctx.astype(np.int64) >> 7) << 15
    flip = rng.random((n, m)) < 0.01
    sym = np.where(flip, sym ^ 0x8000, sym)
    return np.where(rng.random((n, m)) < 0.001, sym & 0x8000, sym).astype(np.uint16), ctx


@pytest.mark.parametrize("n,m,scales,spread", [
    (64, 1024, 2, 20),          # counted
    (64, 1024, 64, 20),         # too few elements per scale
    (64, 1024, 1, 30000),       # too wide
    (300, 256, 3, 12),          # stretches of rows that end inside a scale
    (20, 9000, 1, 40),          # rows of three pieces, the last one shorter
    (33, 1022, 1, 40),          # rows that are not fours: the general way
    (5000, 64, 5, 16),
])
def test_fp8_per_row(n, m, scales, spread):
    sym, ctx = _weight(n, m, spread, n + m)
    sc = (0x3F00 + np.arange(n) % scales).astype(np.uint16)
    built = MPServe_cuda.huffman_build_fp8_decode_tables(torch.from_numpy(sym).view(torch.bfloat16).cuda(), torch.from_numpy(ctx).cuda(),
                                                         torch.from_numpy(sc).cuda(), max_len=7, threads_per_block=64)
    _same(built, orc.build_fp8(sym, ctx, sc, 7, 64))


@pytest.mark.parametrize("bs0,bs1,scales", [(1, 128, 3), (16, 64, 2), (128, 128, 1)])
def test_int4_blocks(bs0, bs1, scales):
    n, m = 128, 512
    sym, ctx = _weight(n, m, 30, bs0 + bs1)
    ctx &= 0x0F
    sc = (0x3C00 + np.arange((n // bs0) * (m // bs1)) % scales).astype(np.uint16).reshape(n // bs0, m // bs1)
    w = torch.from_numpy(sym).view(torch.bfloat16).cuda(), torch.from_numpy(ctx).cuda(), torch.from_numpy(sc).cuda()
    built = MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables_by_scale(*w, max_len=11, threads=64, group_cap=50)
    _same(built, orc.build_awq_by_scale(sym, ctx, sc, 11, 64, 50))
