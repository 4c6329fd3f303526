"""The order that is made for a plan's items, against the same rules in numpy: the end of a launch longest first, what comes
before by number, and batches of neighbours with equal tables that are no larger than their share of the work that is left.
Only the row offsets and tables are read, so the tensors here have nothing else."""
import ctypes as C

import numpy as np
import pytest
import torch

from mpserve_b200 import _lib

pytestmark = pytest.mark.gpu

ITEM_STEPS, SORTED_LOAD, MAX_GRAB, GRAB_SLACK = 40, 10, 8, 4


def _made(rows_of, tables, m, k, threads, chains):
    """Batch starts, (tensor, bucket, first sub-stream) and costs of the order for tensors of `m` columns whose buckets have
    `rows_of[t][b]` rows and the context -> table map that `tables[t][b]` numbers."""
    lib = _lib.load()
    descs, keep, prefix = (_lib.BucketTensor * len(rows_of))(), [], [0]
    span = threads * chains
    chunks = -(-k // span)
    for d, rows, table in zip(descs, rows_of, tables):
        B = len(rows)
        ofs = torch.from_numpy(np.concatenate([[0], np.cumsum(rows)]).astype(np.int32)).cuda()
        width = torch.full((B,), m, dtype=torch.int32, device="cuda")
        btab = torch.from_numpy(np.repeat(np.asarray(table, np.int32)[:, None], 256, axis=1)).cuda()
        keep += [ofs, width, btab]
        d.bucket_row_offsets, d.bucket_col_len, d.bucket_table = ofs.data_ptr(), width.data_ptr(), btab.data_ptr()
        d.mode, d.k, d.m, d.num_buckets = 0, k, m, B
        prefix.append(prefix[-1] + B * chunks)
    items = prefix[-1]
    on = torch.frombuffer(bytearray(bytes(descs)), dtype=torch.uint8).cuda()
    prefix_on = torch.tensor(prefix, dtype=torch.int64).cuda()
    order = torch.zeros(lib.mps_bucket_batch_order_bytes(items), dtype=torch.uint8, device="cuda")
    scratch = torch.empty(lib.mps_bucket_batch_order_scratch_bytes(items), dtype=torch.uint8, device="cuda")
    _lib.check(lib.mps_bucket_batch_order(on.data_ptr(), prefix_on.data_ptr(), len(rows_of), items, threads, chains, order.data_ptr(),
                                          order.numel(), scratch.data_ptr(), scratch.numel(), None))
    torch.cuda.synchronize()
    raw = order.cpu().numpy()
    head = ((items + 1) * 4 + 15) // 16 * 16
    return raw[:(items + 1) * 4].view(np.uint32), raw[head:].view(np.uint32).reshape(-1, 4)[:, :3]


def _wanted(rows_of, tables, m, k, threads, chains):
    span, sms = threads * chains, torch.cuda.get_device_properties(0).multi_processor_count
    item, cost, same = [], [], []
    for t, (rows, table) in enumerate(zip(rows_of, tables)):
        for b, (r, tab) in enumerate(zip(rows, table)):
            for first in range(0, k, span):
                steps = max(0, -(-(int(r) * m - first) // k))
                item.append((t, b, first))
                cost.append(steps + ITEM_STEPS if r > 0 else 0)
                same.append((t, tab))
    cost = np.array(cost, np.int64)
    left = cost.sum() - np.cumsum(cost) + cost
    key = np.where(left > SORTED_LOAD * sms * cost.max(), np.iinfo(np.int64).max, cost)
    by = np.argsort(-key, kind="stable")
    cost = cost[by]
    left = cost.sum() - np.cumsum(cost) + cost
    most = np.full(cost.size, MAX_GRAB)
    for _ in range(3):
        most = np.where((most > 1) & (most * GRAB_SLACK * sms * np.maximum(cost, 1) > left), most // 2, most)
    starts, run = [], 0
    for i, j in enumerate(by):
        if i and (same[j] != same[by[i - 1]] or most[i] != most[i - 1]):
            run = i
        if (i - run) % most[i] == 0:
            starts.append(i)
    return starts, np.array(item, np.int64)[by], cost, left


@pytest.mark.parametrize("rows_of,tables,m,k,shape", [
    ([[128] + [5] * 5000], [[7] * 5001], 4096, 1024, (256, 4)),                        # one long bucket among short ones
    ([[128, 128] + [64] * 200 + [5] * 5000], [[7] * 5202], 4096, 1024, (256, 4)),
    ([[5] * 5000 + [128]], [[7] * 5001], 4096, 1024, (256, 4)),
    ([[128] * 3000], [list(range(3000))], 4096, 1024, (256, 4)),                       # no end but the last to sort
    ([[1, 128, 0, 30] * 1024, [17] * 1023], [[1, 1, 2, 2] * 1024, [3] * 1023], 2048, 1024, (256, 4)),
    ([[3, 90] * 700], [[0] * 1400], 1000, 1000, (256, 1)),                             # buckets of four items
    ([[40]], [[0]], 4096, 256, (256, 1)),
])
def test_order_and_batches(rows_of, tables, m, k, shape):
    starts, entries = _made(rows_of, tables, m, k, *shape)
    want, items, cost, left = _wanted(rows_of, tables, m, k, *shape)
    np.testing.assert_array_equal(entries, items)
    n = len(items)
    np.testing.assert_array_equal(starts, want + [n] * (n + 1 - len(want)))
    # (what the rules are for: a batch of several is no more than its share)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for a, e in zip(want, want[1:] + [n]):
        assert e - a == 1 or cost[a:e].sum() * GRAB_SLACK * sms <= left[a]
