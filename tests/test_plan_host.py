"""Host side of a decode launch (no GPU): which tensors get work items, how many, and the launch shape
(`mps_bucket_batch_plan` reads sizes from host descriptors and dereferences no device pointer; without a
device it plans for 148 SMs)."""
import ctypes as C

import pytest

from mpserve_b200 import _lib


@pytest.fixture(autouse=True)
def no_overrides(monkeypatch):
    for name in ("MPS_DECODE_THREADS", "MPS_DECODE_CHAINS", "MPS_DECODE_DIRECT"):
        monkeypatch.delenv(name, raising=False)


def _tensor(n, m, buckets, k, mode=0, group_size=0):
    t = _lib.BucketTensor()
    fake = 0x10000   # never dereferenced by the planner; aligned like anything a CUDA allocator returns
    for name in ("ctx_bytes", "bitstream", "decode_syms", "decode_lens", "bucket_table", "bucket_col_start",
                 "bucket_col_len", "bucket_row_offsets", "row_indices", "group_col_start", "thread_startbit",
                 "bucket_bit_base", "out"):
        setattr(t, name, fake)
    t.bitstream_words, t.num_tables, t.num_rows, t.num_buckets = 1 << 20, buckets * 200, n, buckets
    t.k, t.group_size, t.mode, t.n, t.m = k, group_size, mode, n, m
    return t


def _plan(tensors):
    lib = _lib.load()
    arr = (_lib.BucketTensor * len(tensors))(*tensors)
    prefix = (C.c_int64 * (len(tensors) + 1))()
    threads, chains = C.c_int32(0), C.c_int32(0)
    rc = lib.mps_bucket_batch_plan(arr, len(tensors), prefix, C.byref(threads), C.byref(chains))
    return rc, list(prefix), threads.value, chains.value


def test_whole_model_takes_the_widest_items():
    tensors = [_tensor(4096, 4096, 111, 1024) for _ in range(64)] + [_tensor(14336, 4096, 190, 1024) for _ in range(32)]
    rc, prefix, threads, chains = _plan(tensors)
    assert rc == 0 and (threads, chains) == (256, 4)
    assert prefix[1] - prefix[0] == 111 and prefix[-1] == 64 * 111 + 32 * 190   # one item per bucket


@pytest.mark.parametrize("k,shape,items", [(1024, (256, 1), 128), (2048, (256, 2), 128), (4096, (256, 4), 128),
                                           (8192, (256, 4), 256), (256, (256, 1), 32)])
def test_lone_weight_of_few_buckets(k, shape, items):
    """32 buckets: narrower items while every item still finds an SM of its own; buckets that are several
    items each (more sub-streams than an item holds) are not cut further than that."""
    rc, prefix, threads, chains = _plan([_tensor(4096, 4096, 32, k)])
    assert rc == 0 and (threads, chains) == shape and prefix[1] == items


def test_whole_buckets_are_halved_up_to_the_sm_count_only():
    assert _plan([_tensor(8192, 8192, 129, 1024)])[2:] == (256, 2)   # 129 items at full width: halve once
    assert _plan([_tensor(8192, 8192, 188, 1024)])[2:] == (256, 4)   # more buckets than SMs: full width


def test_tensors_of_tiny_buckets_get_no_items():
    awq_rect = _tensor(4096, 4096, 4096 * 4096 // 128, 256, mode=1)      # one bucket per 128-element group
    small = _tensor(128, 256, 67, 1024)                                  # under one step per sub-stream
    two_steps = _tensor(512, 1024, 171, 1024)                            # 3066 elements per bucket
    five_steps = _tensor(512, 1024, 100, 1024)                           # 5242 elements per bucket
    big = _tensor(4096, 4096, 111, 1024)
    rc, prefix, threads, chains = _plan([big, big, small, two_steps, five_steps])
    assert rc == 0 and (threads, chains) == (256, 4) and prefix == [0, 111, 222, 222, 222, 322]
    lib = _lib.load()
    arr = (_lib.BucketTensor * 1)(awq_rect)
    pre = (C.c_int64 * 2)()
    th, ch = C.c_int32(0), C.c_int32(0)
    assert lib.mps_bucket_batch_plan(arr, 1, pre, C.byref(th), C.byref(ch)) == 0 and pre[1] == 0


@pytest.mark.parametrize("k", [0, -1, 8193])
def test_sub_stream_count_is_checked(k):
    rc, _, _, _ = _plan([_tensor(4096, 4096, 32, k)])
    assert rc == _lib.MPS_ERR_INVALID
    assert b"invalid k" in _lib.load().mps_last_error()


def test_null_pointer_and_mode_mismatch_are_refused():
    t = _tensor(4096, 4096, 32, 1024)
    t.out = None
    assert _plan([t])[0] == _lib.MPS_ERR_INVALID
    by_scale = _tensor(4096, 4096, 462, 256, mode=2, group_size=0)      # by-scale groups need their size
    assert _plan([by_scale])[0] == _lib.MPS_ERR_INVALID


def test_decode_argument_check_takes_finer_sub_streams():
    """The Python-side check of the rectangular decode calls: up to MAX_SUBSTREAMS sub-streams per bucket."""
    import torch

    from mpserve_b200 import api

    B = 3
    i32 = lambda n: torch.zeros(n, dtype=torch.int32)
    args = lambda k: (i32(B), i32(B), i32(B + 1), i32(7), torch.zeros((B, k + 1), dtype=torch.uint32),
                      torch.zeros(B + 1, dtype=torch.int64), B)
    assert api._check_rect(*args(1024)) == 1024
    assert api._check_rect(*args(api.MAX_SUBSTREAMS)) == api.MAX_SUBSTREAMS
    with pytest.raises(ValueError, match="invalid k"):
        api._check_rect(*args(api.MAX_SUBSTREAMS + 1))


@pytest.mark.parametrize("n,m,k", [(64, 512, 2048), (9, 1000, 4096), (3, 5, 8192)])
def test_oracle_round_trip_with_the_limit_lifted(n, m, k):
    """The checker of the finer sub-streams: the oracle's layout code takes any sub-stream count once its
    argument check (the reference's, 1024) is lifted, and its decode restores the source."""
    import numpy as np
    import torch

    from mpserve_b200 import workloads as wl
    from oracle import oracle as orc

    c = wl.quantize_fp8(wl.random_weight(n, m, 5 + n, "normal"), "channel")
    bits = c.bf16.view(torch.uint16).numpy()
    with pytest.raises(ValueError, match="1024"):
        orc.build_fp8(bits, c.fp8_u8.numpy(), c.scales_u16.numpy(), 7, k)
    orc.set_substream_limit(8192)
    try:
        art = orc.build_fp8(bits, c.fp8_u8.numpy(), c.scales_u16.numpy(), 7, k)
    finally:
        orc.set_substream_limit(1024)
    assert art["bucket_thread_startbit_u32"].shape[1] == k + 1
    np.testing.assert_array_equal(orc.decode_fp8(c.fp8_u8.numpy(), art, n, m), bits)


def _shape(t):
    kernel, threads, chains = C.c_int32(-1), C.c_int32(0), C.c_int32(0)
    assert _lib.load().mps_decode_bucket_shape(C.byref(t), C.byref(kernel), C.byref(threads), C.byref(chains)) == 0
    return ("direct", "narrow", "wide")[kernel.value], threads.value, chains.value


@pytest.mark.parametrize("n,m,buckets,k,shape", [
    (512, 2048, 285, 1024, ("wide", 256, 4)),       # 3 steps a sub-stream: four items a bucket would stage its tables four times
    (1024, 4096, 370, 1024, ("wide", 256, 4)),      # 11
    (2048, 4096, 400, 1024, ("narrow", 256, 1)),    # 20
    (2048, 4096, 512, 1024, ("narrow", 256, 1)),    # 16: the line
    (2048, 4096, 513, 1024, ("wide", 256, 4)),
    (512, 1024, 281, 512, ("narrow", 256, 1)), (14336, 4096, 814, 256, ("narrow", 256, 1))])
def test_by_scale_tensors_by_themselves(n, m, buckets, k, shape):
    assert _shape(_tensor(n, m, buckets, k, mode=2, group_size=128)) == shape


def test_rows_that_bulk_copies_cannot_bring_in():
    assert _shape(_tensor(8000, 3000, 132, 1024)) == ("narrow", 256, 1)
    assert _shape(_tensor(8000, 3001, 132, 1024)) == ("wide", 256, 1)
    assert _shape(_tensor(8000, 3008, 170, 1024)) == ("wide", 256, 4)
    assert _shape(_tensor(1000, 1000, 168, 1024, mode=1)) == ("wide", 256, 4)     # INT4, 5 steps
    assert _shape(_tensor(1000, 1001, 168, 1024, mode=1))[1:] == (256, 1)
    assert _shape(_tensor(128, 256, 67, 1024))[0] == "direct"


def _fp8(n, m, buckets, k, width=None):
    t = _tensor(n, m, buckets, k)
    if width:      # rectangular scale blocks: every bucket lists its own rows
        t.num_rows = n * (m // width)
    return t


@pytest.mark.parametrize("tensor,kernel", [
    (_fp8(4000, 1024, 110, 256), "narrow"), (_fp8(4000, 1040, 110, 256), "wide"),     # 512 steps at most, 520
    (_fp8(241, 5632, 51, 256), "wide"), (_fp8(64, 2048, 36, 256), "narrow"),          # few rows, fewer steps
    (_fp8(4096, 4096, 1024, 256, 128), "narrow"),                                     # blocks of 128 columns, 64 steps
    (_fp8(4000, 1024, 110, 255), "wide"), (_fp8(4000, 1024, 110, 192), "narrow"), (_fp8(4000, 4096, 93, 128), "narrow"),
    (_fp8(4096, 14336, 32, 1024), "narrow"), (_fp8(2047, 3000, 79, 256), "narrow"), (_fp8(2047, 3001, 79, 256), "wide"),
    (_tensor(4096, 4096, 454, 100, mode=2, group_size=128), "wide"), (_tensor(4096, 4096, 454, 104, mode=2, group_size=128), "narrow"),
    (_tensor(4096, 4096, 454, 250, mode=2, group_size=128), "narrow"), (_tensor(1000, 1001, 168, 64, mode=1), "wide"),
    (_tensor(1000, 1001, 168, 128, mode=1), "narrow"), (_tensor(8192, 4096, 207, 255, mode=1), "narrow")])
def test_kernel_of_items_of_256(tensor, kernel):
    assert _shape(tensor)[0] == kernel and _shape(tensor)[1:] == (256, 1)


L8 = [(4096, 4096, 111), (1024, 4096, 92), (1024, 4096, 92), (4096, 4096, 111), (14336, 4096, 190), (14336, 4096, 190), (4096, 14336, 107)]


@pytest.mark.parametrize("tensors,kernel", [
    ([_fp8(n, m, b, 256) for n, m, b in L8], "wide"), ([_fp8(n, m, b, 128) for n, m, b in L8], "narrow"),
    ([_fp8(n, m, n * m // 16384, 256, 128) for n, m, _ in L8], "narrow"),              # 128 x 128 blocks
    ([_fp8(512, 512, 87, 256)] * 16, "narrow"), ([_fp8(4096, 768, 118, 256)] * 4, "wide"),
    ([_fp8(4096, 3000, 100, 256)] * 2 + [_fp8(4096, 4096, 111, 256)], "narrow"),       # what most elements want
    ([_fp8(4096, 3001, 100, 256)] * 2 + [_fp8(4096, 3000, 111, 256)], "wide"),
    ([_tensor(4096, 4096, 454, 256, mode=2, group_size=128)] * 4, "narrow"),
    ([_fp8(4096, 4096, 32, 1024)], "narrow"), ([_fp8(4096, 4096, 32, 255)], "wide")])
def test_kernel_of_a_plan(tensors, kernel):
    """Plans of items of 256 sub-streams go to the kernel that most of their elements want."""
    lib = _lib.load()
    rc, _, threads, chains = _plan(tensors)
    assert rc == 0 and (threads, chains) == (256, 1)
    arr = (_lib.BucketTensor * len(tensors))(*tensors)
    assert ("direct", "narrow", "wide")[lib.mps_bucket_batch_kernel(arr, len(tensors), threads, chains)] == kernel
    assert lib.mps_bucket_batch_kernel(arr, len(tensors), 256, 4) == 2
