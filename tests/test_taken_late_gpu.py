"""Lone tensors on either side of the lines between the forms of a launch: items taken at the start of the one before or late, a
CTA per item or several, and by-scale buckets by number or longest first."""
import numpy as np
import pytest
import torch

import MPServe_cuda
from tests.test_item_order_gpu import KEYS, SMS, _weight

pytestmark = pytest.mark.gpu

BY_SCALE_KEYS = ("bitstream_u64", "decode_syms_u16", "decode_lens_u8", "bucket_table_i32", "bucket_group_offsets_i32", "group_rows_i32",
                 "group_col_start_i32", "bucket_thread_startbit_u32", "bucket_bit_base_i64")
LATE = SMS * 8 // 5


@pytest.mark.parametrize("buckets", [SMS, SMS + 1, LATE, LATE + 1, 2 * SMS + 1])
@pytest.mark.parametrize("k,chains,narrow", [(256, 1, 0), (256, 1, 1), (512, 2, 0), (1024, 4, 0), (1024, 2, 0)])
def test_fp8(buckets, k, chains, narrow, monkeypatch):
    for name, value in (("DIRECT", 0), ("THREADS", 256), ("CHAINS", chains), ("NARROW", narrow)):
        monkeypatch.setenv("MPS_DECODE_" + name, str(value))
    sym, ctx, art = _weight(buckets, 2048, k, buckets + k, 12)
    for _ in range(2):      # (the second launch finds the queue as the first left it)
        out = MPServe_cuda.huffman_decode_fp8(ctx, *[art[key] for key in KEYS], ctx.shape[0], 2048, 7)
        assert torch.equal(out.view(torch.uint16), sym)


@pytest.mark.parametrize("buckets,m", [(300, 1024), (300, 2048), (300, 2560), (300, 4096), (149, 2560), (149, 1024)])
def test_fp8_four_chains(buckets, m, monkeypatch):
    """Items of six to twenty-six steps on average, on either side of the sixteen from which on they are taken late."""
    for name, value in (("DIRECT", 0), ("THREADS", 256), ("CHAINS", 4)):
        monkeypatch.setenv("MPS_DECODE_" + name, str(value))
    sym, ctx, art = _weight(buckets, m, 1024, buckets + m, 12)
    for _ in range(2):
        out = MPServe_cuda.huffman_decode_fp8(ctx, *[art[key] for key in KEYS], ctx.shape[0], m, 7)
        assert torch.equal(out.view(torch.uint16), sym)


@pytest.mark.parametrize("n,m,k", [(1536, 1664, 1024), (1536, 1664, 900), (1536, 1664, 256)])
def test_fp8_blocks(n, m, k):
    """A scale per block of 128 x 128, contexts with more symbols than table slots among them."""
    rng = np.random.default_rng(k)
    scale = torch.from_numpy((0x2000 + rng.integers(0, 40, (n // 128, m // 128))).astype(np.uint16)).cuda()
    ctx = torch.from_numpy(rng.integers(0, 200, (n, m)).astype(np.uint8)).cuda()
    sym = torch.from_numpy((0x3C00 + np.where(ctx.cpu().numpy() == 9, rng.integers(0, 600, (n, m)), rng.integers(0, 11, (n, m)))).astype(np.uint16)).cuda()
    art = MPServe_cuda.huffman_build_fp8_decode_tables(sym.view(torch.bfloat16), ctx, scale, max_len=7, threads_per_block=k)
    for _ in range(2):
        out = MPServe_cuda.huffman_decode_fp8(ctx, *[art[key] for key in KEYS], n, m, 7)
        assert torch.equal(out.view(torch.uint16), sym)


def _by_scale(n, m, buckets, k):
    rng = np.random.default_rng(n + buckets + k)
    groups = n * (m // 128)
    scale = np.concatenate([np.arange(buckets), (buckets * rng.random(groups - buckets) ** 3).astype(np.int64)])
    scale = (0x2000 + rng.permutation(scale)).astype(np.uint16).reshape(n, -1)
    ctx = torch.from_numpy(rng.integers(0, 16, (n, m)).astype(np.uint8)).cuda()
    sym = torch.from_numpy((0x3C00 + rng.integers(0, 30, (n, m))).astype(np.uint16)).cuda()
    art = MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables_by_scale(sym.view(torch.bfloat16), ctx, torch.from_numpy(scale).cuda(),
                                                                            max_len=11, threads=k, group_cap=1 << 20)
    assert art["bucket_table_i32"].shape[0] == buckets
    return sym, ctx, art


# 2 * SMS CTAs, a load of 256 steps for each: 32 * 256 * 2 * SMS elements are 1184 rows of 2048
@pytest.mark.parametrize("n,buckets,k", [(1184, 2 * SMS, 32), (1184, 2 * SMS + 1, 32), (1183, 2 * SMS + 1, 32), (1184, 1792, 32), (1184, 1793, 32),
                                         (1184, 700, 300), (100, SMS + 1, 1024), (60, LATE + 1, 1024)])
def test_by_scale(n, buckets, k):
    sym, ctx, art = _by_scale(n, 2048, buckets, k)
    for _ in range(2):
        out = MPServe_cuda.huffman_decode_awq_int4_bucket_by_scale(ctx, *[art[key] for key in BY_SCALE_KEYS], n, 2048, 11, 128)
        assert torch.equal(out.view(torch.uint16), sym)
