"""Bucket lists made on the GPU are those that the host code makes from the same scales."""
import numpy as np
import pytest
import torch

import MPServe_cuda
from mpserve_b200 import _lib, encoder
from mpserve_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _device_lists(scales, mode, n, nb1, sb0, size, cap, with_cols):
    lib = _lib.load()
    d = torch.from_numpy(scales).cuda()
    out = encoder._sorted_lists(lib, d, mode, n, nb1, sb0, size, cap, with_cols, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return [None if t is None else t.cpu().numpy() for t in out]


def _scales(count, distinct, seed):
    return np.random.default_rng(seed).choice(np.array([0, 1, 0x3C00, 0x7FFF, 0x8000, 0xFFFF], np.uint16) if distinct == 6 else
                                              np.arange(distinct, dtype=np.uint16), count).astype(np.uint16)


@pytest.mark.parametrize("n,distinct", [(1, 1), (127, 1), (128, 1), (129, 2), (1000, 6), (70000, 65535)])
@pytest.mark.parametrize("mode", [0, 1])
def test_rows_by_scale(n, distinct, mode):
    m = 48
    s = _scales(1 if mode == 0 else n, distinct, n)
    scale, ofs, rows, cols = _device_lists(s, mode, n, 1, 1, m, 128, False)
    want = encoder.rect_buckets(s, mode, n, m, n, 1, 1, m)
    for got, ref in zip((scale, ofs, rows), want):
        np.testing.assert_array_equal(got, ref)
        assert got.dtype == ref.dtype
    assert cols is None


@pytest.mark.parametrize("nb0,nb1,sb0,distinct", [(1, 1, 1, 1), (3, 5, 1, 2), (3, 5, 4, 6), (400, 32, 1, 300), (7, 1, 9, 3)])
@pytest.mark.parametrize("cap", [1, 7, 1024, 1 << 40])
def test_groups_by_scale(nb0, nb1, sb0, distinct, cap):
    n, sb1 = nb0 * sb0, 16
    s = _scales(nb0 * nb1, distinct, nb0 + nb1).reshape(nb0, nb1)
    got = _device_lists(s, 2, n, nb1, sb0, sb1, cap, True)
    want = encoder.ragged_buckets(s, 2, n, nb1 * sb1, nb1, sb0, sb1, cap)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
        assert a.dtype == b.dtype


@pytest.mark.parametrize("cap", [2**31, 2**32, 2**63, 2**64])
def test_group_cap_of_any_size(cap):
    """Caps beyond 32 and 64 bits are caps beyond the number of groups."""
    c = wl.quantize_awq(wl.random_weight(64, 512, 5, "normal"), 128)
    w = c.bf16, c.int4_u8, c.scales_u16
    want = MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables_by_scale(*w, max_len=11, threads=64, group_cap=256)
    got = MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables_by_scale(*w, max_len=11, threads=64, group_cap=cap)
    assert set(got) == set(want) and all(torch.equal(got[key].view(torch.uint8), want[key].view(torch.uint8)) for key in want)
