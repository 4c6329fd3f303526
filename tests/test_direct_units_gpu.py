"""The per-sub-stream decoder where buckets are many and smaller than their sub-streams: units of 256 sub-streams and of whole
buckets on either side of the line between them, buckets larger than the average among them, up to more elements than
sub-streams; and short sub-streams of several symbols in more units than the grid has warps."""
import numpy as np
import pytest
import torch

import MPServe_cuda
from tests.test_item_order_gpu import KEYS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [256, 300, 512, 1024])
@pytest.mark.parametrize("m,shared", [(255, 0), (256, 0), (257, 0), (200, 40), (130, 60)])
def test_fp8_rows(m, shared, k):
    """Some 2400 scales of a row each but for `shared`, which have up to seven."""
    rng = np.random.default_rng(m + k)
    scale = np.concatenate([np.arange(2400), np.repeat(rng.integers(0, 2400, shared), rng.integers(1, 7, shared))]).astype(np.uint16)
    rng.shuffle(scale)
    n = scale.size
    ctx = torch.from_numpy(rng.integers(0, 4, (n, m)).astype(np.uint8)).cuda()
    sym = torch.from_numpy((0x3C00 + rng.integers(0, 40, (n, m))).astype(np.uint16)).cuda()
    art = MPServe_cuda.huffman_build_fp8_decode_tables(sym.view(torch.bfloat16), ctx, torch.from_numpy(scale).cuda(), max_len=7,
                                                       threads_per_block=k)
    out = MPServe_cuda.huffman_decode_fp8(ctx, *[art[key] for key in KEYS], n, m, 7)
    assert torch.equal(out.view(torch.uint16), sym)


@pytest.mark.parametrize("n,m,k", [(128, 2560, 512), (128, 2560, 1000), (128, 2432, 1024), (300, 2048, 256), (64, 4096, 1024), (1024, 4096, 64),
                                   (600, 2048, 100)])
def test_int4_groups(n, m, k):
    """A bucket per group of 128; some contexts with more symbols than the table has slots."""
    rng = np.random.default_rng(n + k)
    ctx = torch.from_numpy(rng.integers(0, 16, (n, m)).astype(np.uint8)).cuda()
    sym = torch.from_numpy((0x3C00 + np.where(ctx.cpu().numpy() == 3, rng.integers(0, 9000, (n, m)), rng.integers(0, 90, (n, m)))).astype(np.uint16)).cuda()
    scale = torch.from_numpy((0x3000 + rng.integers(0, 20, (n, m // 128))).astype(np.uint16)).cuda()
    art = MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables(sym.view(torch.bfloat16), ctx, scale, max_len=11, threads_per_block=k)
    out = MPServe_cuda.huffman_decode_awq_int4_bucket(ctx, *[art[key] for key in KEYS], n, m, 11)
    assert torch.equal(out.view(torch.uint16), sym)
