"""The decode kernel for items of 256 sub-streams where it changes its form: steps that end inside a block and inside a
stage, buckets of fewer sub-streams than an item, several items per bucket, rows that come in eights and rows that do
not, rows shorter than a step, buckets of more groups than shared memory holds, and codes with 16 raw bits: none, rare,
almost every symbol (the bitstream then runs through its ring five times as fast), and in stretches."""
import numpy as np
import pytest
import torch

import MPServe_cuda
from mpserve_b200 import util
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

BY_SCALE = ("bitstream_u64", "decode_syms_u16", "decode_lens_u8", "bucket_table_i32", "bucket_group_offsets_i32", "group_rows_i32",
            "group_col_start_i32", "bucket_thread_startbit_u32", "bucket_bit_base_i64")


def _weight(n, m, contexts, esc, seed):
    """esc: None, "rare" (one symbol in 500 is one of thousands), "all" (every symbol is), or "stretches"."""
    rng = np.random.default_rng(seed)
    ctx = rng.integers(0, contexts, (n, m)).astype(np.uint8)
    sym = 0x3C00 + ctx.astype(np.int64) * 16 + np.minimum(rng.geometric(0.4, (n, m)), 15)
    share = {None: 0.0, "rare": 0.002, "all": 1.0}.get(esc)
    wild = rng.random((n, m)) < share if share is not None else (np.arange(n * m).reshape(n, m) // 9000) % 2 == 0
    return np.where(wild, rng.integers(0x4000, 0x7F00, (n, m)), sym).astype(np.uint16), ctx


@pytest.mark.parametrize("esc", [None, "rare", "all", "stretches"])
@pytest.mark.parametrize("n,m,k", [(1, 1, 1), (3, 40, 16), (16, 1000, 256), (9, 1003, 256), (130, 264, 256), (40, 520, 1024), (2, 100, 37),
                                   (64, 248, 250)])
def test_fp8(n, m, k, esc, monkeypatch):
    monkeypatch.setenv("MPS_DECODE_DIRECT", "0")
    monkeypatch.setenv("MPS_DECODE_THREADS", "256")
    monkeypatch.setenv("MPS_DECODE_CHAINS", "1")
    sym, ctx = _weight(n, m, 5, esc, n * m + k)
    art = orc.build_fp8(sym, ctx, np.full(n, 0x3F80, np.uint16), 7, k)
    d = util.artifacts_to_device(art, torch.device("cuda:0"))
    got = util.bf16_bits(MPServe_cuda.huffman_decode_fp8(*util.decode_fp8_args(torch.from_numpy(ctx).cuda(), d, n, m, 7)))
    np.testing.assert_array_equal(got, sym)


@pytest.mark.parametrize("esc", [None, "rare", "all", "stretches"])
@pytest.mark.parametrize("n,groups,size,k,cap", [(5, 2, 128, 256, 1024), (300, 4, 128, 256, 1024), (300, 5, 128, 256, 2000), (64, 3, 64, 100, 50),
                                                 (33, 2, 36, 256, 1024), (200, 1, 24, 1024, 300), (1, 1, 8, 256, 1)])
def test_by_scale(n, groups, size, k, cap, esc, monkeypatch):
    monkeypatch.setenv("MPS_DECODE_DIRECT", "0")
    m = groups * size
    sym, ctx = _weight(n, m, 16, esc, n + size)
    scale = (0x3C00 + (np.arange(n * groups) % 7 == 0)).astype(np.uint16).reshape(n, groups)
    art = orc.build_awq_by_scale(sym, ctx, scale, 11, k, cap)
    d = util.artifacts_to_device(art, torch.device("cuda:0"))
    out = MPServe_cuda.huffman_decode_awq_int4_bucket_by_scale(torch.from_numpy(ctx).cuda(), *[d[key] for key in BY_SCALE], n, m, 11, size)
    np.testing.assert_array_equal(util.bf16_bits(out), sym)


def test_by_scale_context_without_a_table(monkeypatch):
    """A context that a bucket has no table for reads as a code of 11 bits followed by 16 raw ones, as in the oracle."""
    monkeypatch.setenv("MPS_DECODE_DIRECT", "0")
    n, m = 40, 256
    sym, ctx = _weight(n, m, 16, None, 3)
    art = orc.build_awq_by_scale(sym, ctx, np.full((n, 2), 0x3C00, np.uint16), 11, 64, 1024)
    art["bucket_table_i32"][:, 5] = -1
    # (what follows such a symbol is decoded from a wrong place: words to run into)
    art["bitstream_u64"] = np.concatenate([art["bitstream_u64"], np.zeros(256, np.uint64)])
    d = util.artifacts_to_device(art, torch.device("cuda:0"))
    out = MPServe_cuda.huffman_decode_awq_int4_bucket_by_scale(torch.from_numpy(ctx).cuda(), *[d[key] for key in BY_SCALE], n, m, 11, 128)
    np.testing.assert_array_equal(util.bf16_bits(out), orc.decode_awq_by_scale(ctx, art, n, m, 128))


@pytest.fixture
def wide_one_chain(monkeypatch):
    """Items of 256 sub-streams through the wide kernel, one chain per thread: what decodes long sub-streams of 256 and
    rows that are no whole 8-byte pieces."""
    for name, value in (("DIRECT", "0"), ("THREADS", "256"), ("CHAINS", "1"), ("NARROW", "0")):
        monkeypatch.setenv("MPS_DECODE_" + name, value)


@pytest.mark.parametrize("esc", [None, "rare", "all", "stretches"])
@pytest.mark.parametrize("n,m,k", [
    (1, 1, 1), (9, 1003, 256), (64, 250, 1024), (200, 3, 256), (64, 64, 1),
    (128, 1280, 256),      # whole steps per row, more than 512 of them
    (130, 1040, 256),      # steps that split over two rows, a ragged last one, two buckets
    (100, 2048, 1024),     # four items per bucket
    (64, 400, 256), (512, 48, 32), (256, 64, 256), (40, 520, 1024)])
def test_fp8_wide_kernel_with_one_chain(n, m, k, esc, wide_one_chain):
    sym, ctx = _weight(n, m, 5, esc, n * m + k)
    art = orc.build_fp8(sym, ctx, np.full(n, 0x3F80, np.uint16), 7, k)
    d = util.artifacts_to_device(art, torch.device("cuda:0"))
    got = util.bf16_bits(MPServe_cuda.huffman_decode_fp8(*util.decode_fp8_args(torch.from_numpy(ctx).cuda(), d, n, m, 7)))
    np.testing.assert_array_equal(got, sym)


@pytest.mark.parametrize("esc", [None, "rare", "all"])
@pytest.mark.parametrize("n,m,k", [(128, 1024, 256), (60, 1001, 256), (130, 272, 256)])
def test_awq_wide_kernel_with_one_chain(n, m, k, esc, wide_one_chain):
    sym, ctx = _weight(n, m, 16, esc, n + m)
    art = orc.build_awq_bucket(sym, ctx, np.full(n, 0x3F80, np.uint16), 11, k)
    keys = ("bitstream_u64", "decode_syms_u16", "decode_lens_u8", "bucket_table_i32", "bucket_col_start_i32",
            "bucket_col_len_i32", "bucket_row_offsets_i32", "row_indices_i32", "bucket_thread_startbit_u32", "bucket_bit_base_i64")
    d = util.artifacts_to_device(art, torch.device("cuda:0"))
    out = MPServe_cuda.huffman_decode_awq_int4_bucket(torch.from_numpy(ctx).cuda(), *[d[key] for key in keys], n, m, 11)
    np.testing.assert_array_equal(util.bf16_bits(out), sym)


@pytest.mark.parametrize("kernel", [None, "0", "1"])
@pytest.mark.parametrize("shapes,k", [([(300, 768), (64, 520), (130, 1003)], 256), ([(200, 400), (64, 1024)], 96), ([(40, 520), (129, 264)], 255)])
def test_plans_of_narrow_items(shapes, k, kernel, monkeypatch):
    """Tensors of several kinds in one launch of 256 x 1 items: through the plan's own choice and through either kernel."""
    from mpserve_b200.api import BucketDecodePlan

    if kernel is not None:
        monkeypatch.setenv("MPS_DECODE_NARROW", kernel)
    entries, want = [], []
    for i, (n, m) in enumerate(shapes):
        sym, ctx = _weight(n, m, 5, "rare" if i else None, n + m)
        art = orc.build_fp8(sym, ctx, np.full(n, 0x3F80, np.uint16), 7, k)
        entries.append((torch.from_numpy(ctx).cuda(), util.artifacts_to_device(art, torch.device("cuda:0")), None))
        want.append(sym)
    plan = BucketDecodePlan(entries)
    assert (plan.threads, plan.chains) == (256, 1)
    for out, sym in zip(plan.decode(), want):
        np.testing.assert_array_equal(util.bf16_bits(out), sym)
