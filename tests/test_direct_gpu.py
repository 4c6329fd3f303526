"""The per-sub-stream decoder at the sizes where it changes its form: sub-streams of one symbol (no more elements than
sub-streams) and of more, units that end inside a pass of a warp, one row and several, and contexts with more symbols
than table slots, so that ESC codes with their 16 raw bits occur among single-symbol sub-streams."""
import numpy as np
import pytest
import torch

from mpserve_b200 import util
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _weights(n, m, contexts, symbols, seed):
    """Random patterns: every context sees up to ``symbols`` different ones, so ESC codes follow from the sizes."""
    rng = np.random.default_rng(seed)
    ctx = rng.integers(0, contexts, (n, m)).astype(np.uint8)
    sym = (0x3C00 + rng.integers(0, symbols, (n, m)) * 3).astype(np.uint16)
    return sym, ctx


@pytest.mark.parametrize("n,m,k", [(1, 1, 1), (1, 31, 32), (3, 129, 512), (1, 1024, 1024), (2, 500, 1000), (5, 333, 1024),
                                   (4, 128, 256), (7, 130, 255), (130, 64, 200)])
def test_fp8_small_buckets(n, m, k, monkeypatch):
    import MPServe_cuda

    monkeypatch.setenv("MPS_DECODE_DIRECT", "1")
    sym, ctx = _weights(n, m, 2, 300, n * m + k)
    scale = np.full(n, 0x3F80, np.uint16)
    art = orc.build_fp8(sym, ctx, scale, 7, k)
    d = util.artifacts_to_device(art, torch.device("cuda:0"))
    got = util.bf16_bits(MPServe_cuda.huffman_decode_fp8(*util.decode_fp8_args(torch.from_numpy(ctx).cuda(), d, n, m, 7)))
    np.testing.assert_array_equal(got, orc.decode_fp8(ctx, art, n, m))
    np.testing.assert_array_equal(got, sym)


@pytest.mark.parametrize("n,m,k,symbols", [(3, 128, 256, 40), (3, 128, 256, 4000), (40, 256, 128, 4000), (2, 128, 100, 300),
                                           (1, 8192, 1024, 6000), (300, 128, 1024, 6000)])
def test_awq_small_buckets(n, m, k, symbols, monkeypatch):
    import MPServe_cuda

    monkeypatch.setenv("MPS_DECODE_DIRECT", "1")
    sym, ctx = _weights(n, m, 1 if symbols > 2048 else 16, symbols, n + m + k)
    scale = (0x3C00 + np.arange(n * (m // 128)) % 2).astype(np.uint16).reshape(n, m // 128)
    art = orc.build_awq_bucket(sym, ctx, scale, 11, k)
    keys = ("bitstream_u64", "decode_syms_u16", "decode_lens_u8", "bucket_table_i32", "bucket_col_start_i32",
            "bucket_col_len_i32", "bucket_row_offsets_i32", "row_indices_i32", "bucket_thread_startbit_u32", "bucket_bit_base_i64")
    d = util.artifacts_to_device(art, torch.device("cuda:0"))
    out = MPServe_cuda.huffman_decode_awq_int4_bucket(torch.from_numpy(ctx).cuda(), *[d[key] for key in keys], n, m, 11)
    got = util.bf16_bits(out)
    np.testing.assert_array_equal(got, orc.decode_awq_bucket(ctx, art, n, m))
    np.testing.assert_array_equal(got, sym)


def _decode_each(decode, monkeypatch):
    """What the direct kernel, the one for items of 256 sub-streams and the wide one (two shapes) return."""
    for direct, threads, chains in (("1", "0", "0"), ("0", "256", "1"), ("0", "256", "4"), ("0", "512", "1")):
        monkeypatch.setenv("MPS_DECODE_DIRECT", direct)
        monkeypatch.setenv("MPS_DECODE_THREADS", threads)
        monkeypatch.setenv("MPS_DECODE_CHAINS", chains)
        yield (direct, threads, chains), util.bf16_bits(decode())


@pytest.mark.parametrize("n,m,k", [(1, 1024, 1024), (8, 128, 1024), (1, 700, 1000), (3, 1024, 1024)])
def test_fp8_bare_esc(n, m, k, monkeypatch):
    """A symbol without a code of its own that equals the ESC symbol (the smallest one without a code) is written as the
    ESC code alone; a decoder reads the 16 bits that follow, whatever they are, in every kernel."""
    import MPServe_cuda

    sym, ctx = _weights(n, m, 1, 300, n * m + k)
    sym[n // 2, m // 2] = 0
    art = orc.build_fp8(sym, ctx, np.full(n, 0x3F80, np.uint16), 7, k)
    want = orc.decode_fp8(ctx, art, n, m)
    assert want[n // 2, m // 2] != 0, "case was meant to contain a bare ESC code"
    d = util.artifacts_to_device(art, torch.device("cuda:0"))
    args = util.decode_fp8_args(torch.from_numpy(ctx).cuda(), d, n, m, 7)
    for which, got in _decode_each(lambda: MPServe_cuda.huffman_decode_fp8(*args), monkeypatch):
        np.testing.assert_array_equal(got, want, err_msg=str(which))


@pytest.mark.parametrize("n,m,k", [(300, 128, 256), (2500, 128, 128), (20, 2048, 1024)])
def test_awq_bare_esc(n, m, k, monkeypatch):
    import MPServe_cuda

    sym, ctx = _weights(n, m, 1, 6000, n + m + k)
    sym[n // 2, m // 2] = 0
    scale = (0x3C00 + np.arange(n * (m // 128)) % 2).astype(np.uint16).reshape(n, m // 128)
    art = orc.build_awq_bucket(sym, ctx, scale, 11, k)
    want = orc.decode_awq_bucket(ctx, art, n, m)
    assert want[n // 2, m // 2] != 0, "case was meant to contain a bare ESC code"
    keys = ("bitstream_u64", "decode_syms_u16", "decode_lens_u8", "bucket_table_i32", "bucket_col_start_i32",
            "bucket_col_len_i32", "bucket_row_offsets_i32", "row_indices_i32", "bucket_thread_startbit_u32", "bucket_bit_base_i64")
    d = util.artifacts_to_device(art, torch.device("cuda:0"))
    args = (torch.from_numpy(ctx).cuda(), *[d[key] for key in keys], n, m, 11)
    for which, got in _decode_each(lambda: MPServe_cuda.huffman_decode_awq_int4_bucket(*args), monkeypatch):
        np.testing.assert_array_equal(got, want, err_msg=str(which))


@pytest.mark.parametrize("n,m,k", [(2500, 128, 64), (2500, 128, 33), (40, 128, 64), (40, 128, 128), (2400, 128, 1024)])
def test_awq_shares_of_a_warp(n, m, k, monkeypatch):
    """Few buckets and many, of sub-streams of one symbol and of several: one, two and four sub-streams per lane."""
    import MPServe_cuda

    monkeypatch.setenv("MPS_DECODE_DIRECT", "1")
    sym, ctx = _weights(n, m, 16, 300, n + m + k)
    art = orc.build_awq_bucket(sym, ctx, np.full((n, 1), 0x3C00, np.uint16), 11, k)
    assert art["bucket_table_i32"].shape[0] == n
    keys = ("bitstream_u64", "decode_syms_u16", "decode_lens_u8", "bucket_table_i32", "bucket_col_start_i32",
            "bucket_col_len_i32", "bucket_row_offsets_i32", "row_indices_i32", "bucket_thread_startbit_u32", "bucket_bit_base_i64")
    d = util.artifacts_to_device(art, torch.device("cuda:0"))
    out = MPServe_cuda.huffman_decode_awq_int4_bucket(torch.from_numpy(ctx).cuda(), *[d[key] for key in keys], n, m, 11)
    np.testing.assert_array_equal(util.bf16_bits(out), sym)


@pytest.mark.parametrize("n,m,k", [(2500, 32, 64), (2500, 32, 24), (60, 512, 1024)])
def test_fp8_shares_of_a_warp(n, m, k, monkeypatch):
    import MPServe_cuda

    monkeypatch.setenv("MPS_DECODE_DIRECT", "1")
    sym, ctx = _weights(n, m, 2, 100, n + m + k)
    scale = np.arange(1, n + 1).astype(np.uint16)      # a bucket per row
    art = orc.build_fp8(sym, ctx, scale, 7, k)
    d = util.artifacts_to_device(art, torch.device("cuda:0"))
    got = util.bf16_bits(MPServe_cuda.huffman_decode_fp8(*util.decode_fp8_args(torch.from_numpy(ctx).cuda(), d, n, m, 7)))
    np.testing.assert_array_equal(got, sym)


def test_awq_long_shares_of_a_warp(monkeypatch):
    """More than two million sub-streams of two symbols: a lane takes several after one another."""
    import MPServe_cuda
    from mpserve_b200 import workloads as wl

    monkeypatch.setenv("MPS_DECODE_DIRECT", "1")
    c = wl.quantize_awq(wl.random_weight(2100, 2048, 4, "normal", device="cuda"), 128)
    art = MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables(c.bf16, c.int4_u8, c.scales_u16, max_len=11, threads_per_block=64)
    assert art["bucket_table_i32"].shape[0] * 64 >= 1 << 21
    keys = ("bitstream_u64", "decode_syms_u16", "decode_lens_u8", "bucket_table_i32", "bucket_col_start_i32",
            "bucket_col_len_i32", "bucket_row_offsets_i32", "row_indices_i32", "bucket_thread_startbit_u32", "bucket_bit_base_i64")
    out = MPServe_cuda.huffman_decode_awq_int4_bucket(c.int4_u8, *[art[key] for key in keys], 2100, 2048, 11)
    assert torch.equal(out.view(torch.int16), c.bf16.view(torch.int16))
