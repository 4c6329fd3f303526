"""Codebooks of the GPU sidecar builder at the sizes where its code paths meet: contexts of one symbol, of a warp's
register sort (32), its shared-memory sort, the most a warp takes (128 symbols of a 7-bit table, 512 of a wider
one), the most a CTA takes, the ESC reduction (more symbols than table slots), tables too large for shared
memory (max_len above 11) and all 65536 symbols in one context.  Byte for byte against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _weight(distinct, m, seed):
    """[n, m] symbols and contexts: context c sees ``distinct[c]`` symbols, their counts skewed and with many ties."""
    rng = np.random.default_rng(seed)
    sym, ctx = [], []
    for c, d in enumerate(distinct):
        s = rng.choice(65536, size=d, replace=False)
        counts = 1 + rng.geometric(0.5, size=d) * (rng.random(d) < 0.3) + (rng.pareto(1.0, size=d)).astype(np.int64) % 50
        sym.append(np.repeat(s, counts))
        ctx.append(np.full(int(counts.sum()), c))
    sym, ctx = np.concatenate(sym), np.concatenate(ctx)
    order = rng.permutation(sym.size)
    pad = -sym.size % m
    order = np.concatenate([order, order[:1].repeat(pad)])   # repeats of one element: no new symbol
    return sym[order].astype(np.uint16).reshape(-1, m), ctx[order].astype(np.uint8).reshape(-1, m)


FP8 = [([1, 2, 31, 32, 33, 63, 64, 65, 127, 128], 7), ([129, 130, 1, 300, 5000], 7), ([65536, 3], 7),
       ([1, 2, 3, 4, 5], 1), ([2, 3, 4], 2), ([40, 16, 17], 4), ([4095, 4096, 4097, 512, 513], 12), ([32767, 32769, 7], 15)]
AWQ = [([511, 512, 513, 2047, 2048, 2049, 1, 33], 11), ([65536, 40, 2000], 11), ([64, 65, 128, 129, 600], 6), ([255, 256, 257, 700], 8),
       ([5000, 300], 13)]


def _same(got, want):
    assert set(got) == set(want)
    for key, w in want.items():
        g = got[key].cpu()
        g = g.view(torch.uint16).numpy() if g.dtype == torch.bfloat16 else g.numpy()
        assert g.dtype == w.dtype and np.array_equal(g, w), key


@pytest.mark.parametrize("distinct,L", FP8)
def test_fp8_codebooks_at_their_edges(distinct, L):
    import MPServe_cuda

    sym, ctx = _weight(distinct, 64, 1000 + L)
    scale = np.array([77], dtype=np.uint16)
    got = MPServe_cuda.huffman_build_fp8_decode_tables(torch.from_numpy(sym).view(torch.bfloat16), torch.from_numpy(ctx),
                                                       torch.from_numpy(scale), max_len=L, threads_per_block=96)
    _same(got, orc.build_fp8(sym, ctx, scale, L, 96))


@pytest.mark.parametrize("layout", ["bucket", "by_scale", "shared"])
@pytest.mark.parametrize("distinct,L", AWQ)
def test_awq_codebooks_at_their_edges(distinct, L, layout):
    import MPServe_cuda

    sym, ctx = _weight(distinct, 128, 2000 + L)
    scale = np.array([5], dtype=np.uint16)
    w = torch.from_numpy(sym).view(torch.bfloat16), torch.from_numpy(ctx), torch.from_numpy(scale)
    if layout == "bucket":
        _same(MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables(*w, max_len=L, threads_per_block=64),
              orc.build_awq_bucket(sym, ctx, scale, L, 64))
    elif layout == "by_scale":
        _same(MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables_by_scale(*w, max_len=L, threads=64, group_cap=7),
              orc.build_awq_by_scale(sym, ctx, scale, L, 64, 7))
    else:
        _same(MPServe_cuda.huffman_build_awq_decode_tables(*w, max_len=L), orc.build_awq_shared(sym, ctx, scale, L))
