"""Layout and emission of the GPU sidecar builder where their paths meet: sub-stream counts that are not multiples
of four (one sub-stream per thread), of one sub-stream, of more sub-streams than a CTA holds, rows of odd length,
ragged last steps, buckets too small for code maps in shared memory, symbols spread too widely for them, and
units whose bits do not fit the emit buffer.  Byte for byte against the oracle."""
import numpy as np
import pytest
import torch

from mpserve_b200 import workloads as wl
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _same(got, want):
    assert set(got) == set(want)
    for key, w in want.items():
        g = got[key].cpu()
        g = g.view(torch.uint16).numpy() if g.dtype == torch.bfloat16 else g.numpy()
        assert g.dtype == w.dtype and np.array_equal(g, w), key


@pytest.mark.parametrize("n,m,k,mode,dist", [
    (130, 257, 96, "tensor", "normal"),       # odd rows, one sub-stream per thread
    (128, 1000, 1024, "tensor", "normal"),    # ragged last step
    (256, 512, 3, "tensor", "normal"),
    (64, 4096, 1, "tensor", "normal"),        # one sub-stream of 262144 codes: longer than the emit buffer
    (64, 4096, 4, "channel", "student_t"),
    (70, 4096, 1000, "channel", "normal"),
    (300, 2048, 1024, "channel", "student_t"),
    (37, 20, 512, "channel", "normal"),       # buckets of fewer elements than sub-streams
    (256, 384, 256, "block", "normal"),
    (1024, 2048, 256, "tensor", "normal"),    # units of a bucket share its sub-streams
])
def test_fp8_layout(n, m, k, mode, dist):
    import MPServe_cuda

    c = wl.quantize_fp8(wl.random_weight(n, m, 90 + n + m, dist), mode)
    got = MPServe_cuda.huffman_build_fp8_decode_tables(c.bf16, c.fp8_u8, c.scales_u16, max_len=7, threads_per_block=k)
    _same(got, orc.build_fp8(c.bf16.view(torch.uint16).numpy(), c.fp8_u8.numpy(), c.scales_u16.numpy(), 7, k))


@pytest.mark.parametrize("L", [7, 12])
@pytest.mark.parametrize("n,m,k", [(128, 512, 256), (128, 511, 33)])
def test_fp8_layout_of_scattered_symbols(n, m, k, L):
    """Random patterns under random bytes: maps of 256 x 65536 entries, most elements behind an ESC code of 23 bits or more."""
    import MPServe_cuda

    rng = np.random.default_rng(n + m + L)
    sym = rng.integers(0, 65536, size=(n, m), dtype=np.uint16)
    ctx = rng.integers(0, 3, size=(n, m), dtype=np.uint8) * 100
    scale = np.array([9], dtype=np.uint16)
    got = MPServe_cuda.huffman_build_fp8_decode_tables(torch.from_numpy(sym).view(torch.bfloat16), torch.from_numpy(ctx),
                                                       torch.from_numpy(scale), max_len=L, threads_per_block=k)
    _same(got, orc.build_fp8(sym, ctx, scale, L, k))


@pytest.mark.parametrize("k", [2048, 4096, 8192])
def test_fp8_layout_of_fine_substreams(k):
    from mpserve_b200 import api

    c = wl.quantize_fp8(wl.random_weight(128, 1024, 17, "normal"), "tensor")
    w = c.bf16.cuda(), c.fp8_u8.cuda(), c.scales_u16.cuda()
    art = api.build_fp8_fine_substreams(*w, max_len=7, substreams=k)
    keys = ("bitstream_u64", "decode_syms_u16", "decode_lens_u8", "bucket_table_i32", "bucket_col_start_i32", "bucket_col_len_i32",
            "bucket_row_offsets_i32", "row_indices_i32", "bucket_thread_startbit_u32", "bucket_bit_base_i64")
    out = api.huffman_decode_fp8(w[1], *(art[key] for key in keys), 128, 1024, 7)
    assert torch.equal(out.view(torch.int16), w[0].view(torch.int16))


@pytest.mark.parametrize("n,m,k,cap", [(256, 2048, 256, 1024), (256, 2048, 100, 1024), (256, 2048, 256, 3), (64, 1024, 1024, 1024)])
@pytest.mark.parametrize("one_scale", [False, True])
def test_awq_by_scale_layout(n, m, k, cap, one_scale):
    import MPServe_cuda

    c = wl.quantize_awq(wl.random_weight(n, m, 91 + n + k, "normal"), 128)
    scales = torch.full_like(c.scales_u16.view(torch.int16), 777).view(torch.uint16) if one_scale else c.scales_u16
    got = MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables_by_scale(c.bf16, c.int4_u8, scales, max_len=11, threads=k,
                                                                            group_cap=cap)
    _same(got, orc.build_awq_by_scale(c.bf16.view(torch.uint16).numpy(), c.int4_u8.numpy(), scales.numpy(), 11, k, cap))
