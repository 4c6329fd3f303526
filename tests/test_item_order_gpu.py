"""The order in which work items are taken: longest first, of a lone tensor by the kernel itself, of a plan when it is
made.  Whatever the order, every item is decoded once: sizes around the number of CTAs and the most buckets that a launch
sorts, buckets of several items, and plans whose order is looked at."""
import numpy as np
import pytest
import torch

import MPServe_cuda
from mpserve_b200 import _lib
from mpserve_b200.api import BucketDecodePlan

pytestmark = pytest.mark.gpu

KEYS = ("bitstream_u64", "decode_syms_u16", "decode_lens_u8", "bucket_table_i32", "bucket_col_start_i32", "bucket_col_len_i32",
        "bucket_row_offsets_i32", "row_indices_i32", "bucket_thread_startbit_u32", "bucket_bit_base_i64")
SMS = 148


def _weight(buckets, m, k, seed, most=6):
    """Rows of `buckets` different scales, 1 to `most` rows of each, and their sidecar."""
    rng = np.random.default_rng(seed)
    scale = np.repeat(np.arange(buckets) + 0x2000, rng.integers(1, most + 1, buckets)).astype(np.uint16)
    rng.shuffle(scale)
    n = scale.size
    ctx = torch.from_numpy(rng.integers(0, 4, (n, m)).astype(np.uint8)).cuda()
    sym = torch.from_numpy((0x3C00 + rng.integers(0, 9, (n, m))).astype(np.uint16)).cuda()
    art = MPServe_cuda.huffman_build_fp8_decode_tables(sym.view(torch.bfloat16), ctx, torch.from_numpy(scale).cuda(), max_len=7,
                                                       threads_per_block=k)
    assert art["bucket_table_i32"].shape[0] == buckets
    return sym, ctx, {key: art[key] for key in KEYS}


@pytest.mark.parametrize("buckets,m,k", [(2 * SMS, 1024, 256), (2 * SMS + 1, 1024, 256), (1791, 1024, 256), (1792, 1040, 256),
                                         (1793, 1024, 256), (150, 2048, 512), (77, 4096, 1000)])
def test_lone_tensor(buckets, m, k, monkeypatch):
    monkeypatch.setenv("MPS_DECODE_DIRECT", "0")
    monkeypatch.setenv("MPS_DECODE_THREADS", "256")
    monkeypatch.setenv("MPS_DECODE_CHAINS", "1")
    sym, ctx, art = _weight(buckets, m, k, buckets)
    for _ in range(2):      # (the second launch finds the queue as the first left it)
        out = MPServe_cuda.huffman_decode_fp8(ctx, *[art[key] for key in KEYS], ctx.shape[0], m, 7)
        assert torch.equal(out.view(torch.uint16), sym)


@pytest.mark.parametrize("k,shapes", [(1024, [(200, 4096), (90, 8192)]), (256, [(400, 1024)]), (1024, [(40, 4096), (2500, 3072), (9, 14336)]),
                                      (512, [(300, 2048), (30, 2000)])])
def test_plan(k, shapes):
    weights = [_weight(buckets, m, k, 31 * i + buckets) for i, (buckets, m) in enumerate(shapes)]
    plan = BucketDecodePlan([(ctx, art, None) for _, ctx, art in weights])
    assert plan.total_items > SMS and plan._order is not None
    items = plan.total_items
    raw = plan._order.cpu().numpy()
    head = ((items + 1) * 4 + 15) // 16 * 16
    starts, entries = raw[:(items + 1) * 4].view(np.uint32), raw[head:head + 16 * items].view(np.uint32).reshape(-1, 4)
    # every item once ...
    assert len({tuple(e[:3]) for e in entries.tolist()}) == items
    # ... longest first ...
    prefix = plan._prefix_dev.cpu().numpy()
    offsets = {}
    for i, d in enumerate(plan._descs_host):
        art = next(a for _, _, a in weights if a["bucket_row_offsets_i32"].data_ptr() == d.bucket_row_offsets)
        offsets[i] = (np.diff(art["bucket_row_offsets_i32"].cpu().numpy()), d.m)
    steps = [-(-(int(offsets[t][0][b]) * offsets[t][1] - first) // k) for t, b, first, _ in entries.tolist()]
    assert steps == sorted(steps, reverse=True)
    assert prefix[-1] == items
    # ... in batches that follow one another, of at most eight
    ends = starts[1:].astype(np.int64) - starts[:-1]
    assert starts[0] == 0 and starts[-1] == items and ends.min() >= 0 and ends.max() <= 8
    for _ in range(2):
        for out, (sym, _, _) in zip(plan.decode(), weights):
            assert torch.equal(out.view(torch.uint16), sym)


def test_plan_of_few_items_and_bad_arguments():
    sym, ctx, art = _weight(30, 4096, 1024, 5)
    plan = BucketDecodePlan([(ctx, art, None)])
    assert plan._order is None
    assert torch.equal(plan.decode()[0].view(torch.uint16), sym)
    lib = _lib.load()
    assert lib.mps_bucket_batch_order_bytes(0) == 0 and lib.mps_bucket_batch_order_bytes((1 << 24) + 1) == 0
    buf = torch.empty(1 << 16, dtype=torch.uint8, device="cuda")
    args = (plan._descs_dev.data_ptr(), plan._prefix_dev.data_ptr(), 1, plan.total_items, plan.threads, plan.chains)
    assert lib.mps_bucket_batch_order(*args, buf.data_ptr(), 16, buf.data_ptr(), buf.numel(), None) == _lib.MPS_ERR_WORKSPACE
    assert lib.mps_bucket_batch_order(*args, buf.data_ptr() + 4, 1 << 15, buf.data_ptr(), buf.numel(), None) == _lib.MPS_ERR_INVALID
