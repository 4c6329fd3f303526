"""The builder's C entry points for a caller that makes the bucket lists itself: weights that are not the analyzed ones,
columns cut anywhere, lists that are wrong at first."""
import ctypes as C

import numpy as np
import pytest
import torch

import MPServe_cuda
from mpserve_b200 import _lib
from mpserve_b200.util import bf16_bits

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


class Build:
    """An FP8 weight with one scale, its histogram and codebooks; buckets are (first row, rows, column start, columns)."""

    def __init__(self, sym, ctx, L=7, most_substreams=1 << 16, variant=0):
        self.lib = _lib.load()
        self.n, self.m = sym.shape
        self.L = L
        self.sym, self.ctx, self.scale = _dev(sym), _dev(ctx), _dev(np.array([0x3F80], np.uint16))
        size = self.lib.mps_build_workspace_bytes(sym.size, most_substreams)
        self.ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        self.state = (C.c_ubyte * 256)()
        G, N = C.c_int64(0), C.c_int64(0)
        _lib.check(self.lib.mps_build_analyze(self.state, self.sym.data_ptr(), self.ctx.data_ptr(), self.scale.data_ptr(), 0, 1,
                                              self.n, self.m, self.n, self.m, variant, L, self.ws.data_ptr(), size, None, C.byref(G), C.byref(N)))
        self.G = int(G.value)
        self.key = torch.empty((2, self.G), dtype=torch.uint16, device="cuda")
        if variant != 3:
            self.codebooks()

    def codebooks(self):
        G, TS = self.G, 1 << self.L
        self.syms = torch.empty((G, TS), dtype=torch.uint16, device="cuda")
        self.lens = torch.empty((G, TS // 2), dtype=torch.uint8, device="cuda")
        _lib.check(self.lib.mps_build_codebooks(self.state, self.syms.data_ptr(), self.lens.data_ptr(), self.key[0].data_ptr(),
                                                self.key[1].data_ptr(), None))

    def layout(self, buckets, k, sym=None):
        """The call's status; the lists and what it wrote stay here."""
        B = len(buckets)
        self.B, self.k = B, k
        self.rows = _dev(np.concatenate([np.arange(r, r + h) for r, h, _, _ in buckets]).astype(np.int32))
        self.ofs = _dev(np.cumsum([0] + [h for _, h, _, _ in buckets]).astype(np.int32))
        self.cs = _dev(np.array([c for _, _, c, _ in buckets], np.int32))
        self.cl = _dev(np.array([w for _, _, _, w in buckets], np.int32))
        scales = self.scale.expand(B).contiguous()
        self.btab = torch.empty((B, 256), dtype=torch.int32, device="cuda")
        _lib.check(self.lib.mps_build_bucket_table(self.state, scales.data_ptr(), B, self.btab.data_ptr(), None))
        self.start = torch.empty((B, k + 1), dtype=torch.uint32, device="cuda")
        self.base = torch.empty((B + 1,), dtype=torch.int64, device="cuda")
        total = C.c_int64(0)
        rc = self.lib.mps_build_rect_layout(self.state, (self.sym if sym is None else sym).data_ptr(), self.ctx.data_ptr(),
                                            self.btab.data_ptr(), self.cs.data_ptr(), self.cl.data_ptr(), self.ofs.data_ptr(),
                                            self.rows.data_ptr(), B, k, self.start.data_ptr(), self.base.data_ptr(), None, C.byref(total))
        self.words = (total.value + 63) // 64
        return rc

    def emit(self, k=None, ragged=False):
        self.bits = torch.zeros((max(self.words, 1),), dtype=torch.uint64, device="cuda")
        return self.lib.mps_build_rect_emit(self.state, self.sym.data_ptr(), self.ctx.data_ptr(), self.btab.data_ptr(), self.cs.data_ptr(),
                                            None if ragged else self.cl.data_ptr(), self.ofs.data_ptr(), self.rows.data_ptr(), self.B,
                                            k or self.k, self.start.data_ptr(), self.base.data_ptr(), self.bits.data_ptr(), self.words, None)

    def decoded(self):
        return bf16_bits(MPServe_cuda.huffman_decode_fp8(self.ctx, self.bits, self.syms, self.lens, self.btab, self.cs, self.cl, self.ofs,
                                                         self.rows, self.start, self.base, self.n, self.m, 7))


def _weight(n, m, seed=0):
    """Contexts 0 and 1 with sixteen neighbouring patterns each, not next to one another."""
    rng = np.random.default_rng(seed)
    ctx = rng.integers(0, 2, (n, m)).astype(np.uint8)
    return (0x3C00 + 0x100 * ctx.astype(np.int64) + rng.integers(0, 16, (n, m))).astype(np.uint16), ctx


def test_emit_that_does_not_follow_its_layout():
    """What a layout call leaves behind is read by the emit call of the same buckets and sub-streams only."""
    sym, ctx = _weight(128, 512, 7)
    b = Build(sym, ctx)
    assert b.layout([(0, 128, 0, 256), (0, 128, 256, 256)], 256) == _lib.MPS_OK
    for wrong in (dict(k=255), dict(k=128), dict(k=1024), dict(ragged=True)):
        assert b.emit(**wrong) == _lib.MPS_ERR_INVALID, wrong
        assert b"mps_build_rect_layout" in b.lib.mps_last_error()
    assert b.emit() == _lib.MPS_OK
    np.testing.assert_array_equal(b.decoded(), sym)
    b.codebooks()      # works where the layout call had left its codes
    assert b.emit() == _lib.MPS_ERR_INVALID
    assert b.layout([(0, 128, 0, 256), (0, 128, 256, 256)], 256) == _lib.MPS_OK and b.emit() == _lib.MPS_OK
    np.testing.assert_array_equal(b.decoded(), sym)


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("symbols", [1, 40, 5000])
def test_tables_at_any_address(shared, symbols):
    """Tables of a caller that do not start where torch's allocations do: symbols on an odd multiple of two bytes, lengths on
    an odd byte.  One symbol, those of a warp, and more than the table has slots (a CTA)."""
    rng = np.random.default_rng(symbols)
    sym = (0x3C00 + rng.integers(0, symbols, (96, 512))).astype(np.uint16)
    ctx = rng.integers(0, 2, (96, 512)).astype(np.uint8)
    L, lib = (11, _lib.load()) if shared else (7, _lib.load())
    b = Build(sym, ctx, L, variant=3 if shared else 0)
    rows = 16 if shared else b.G
    nl = (1 << L) if shared else (1 << L) // 2
    lut = torch.full((65536,), -1, dtype=torch.int32, device="cuda")
    lut[0x3F80] = 0
    got = []
    for off in (0, 1):
        syms = torch.zeros((rows * (1 << L) + 1,), dtype=torch.int16, device="cuda")[off:]
        lens = torch.zeros((rows * nl + 1,), dtype=torch.uint8, device="cuda")[off:]
        if shared:
            rc = lib.mps_build_shared_codebooks(b.state, lut.data_ptr(), 1, syms.data_ptr(), lens.data_ptr(), None)
        else:
            rc = lib.mps_build_codebooks(b.state, syms.data_ptr(), lens.data_ptr(), b.key[0].data_ptr(), b.key[1].data_ptr(), None)
        assert rc == _lib.MPS_OK
        got.append((syms[:rows * (1 << L)].cpu(), lens[:rows * nl].cpu()))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert bool(got[0][1].any())


@pytest.mark.parametrize("context,symbol", [(0, 0x3C10), (0, 0x3C1F), (1, 0x3CFF), (0, 0xBC00), (1, 0x3D05)])
def test_symbol_the_analysis_did_not_see(context, symbol):
    """A weight that is not the analyzed one: a symbol outside its context's range is an error, also where another context's
    range begins beside it.  (The last case is inside: it has a code.)"""
    sym, ctx = _weight(128, 512)
    ctx[64, 256] = context
    sym[64, 256] = 0x3C00 + 0x100 * context
    b = Build(sym, ctx)
    assert b.layout([(0, 128, 0, 512)], 256) == _lib.MPS_OK
    other = sym.copy()
    other[64, 256] = symbol
    rc = b.layout([(0, 128, 0, 512)], 256, _dev(other))
    if (context, symbol) == (1, 0x3D05):
        assert rc == _lib.MPS_OK
    else:
        assert rc != _lib.MPS_OK and b"symbol not found" in b.lib.mps_last_error()


@pytest.mark.parametrize("cuts,k", [((0, 129, 512), 256), ((0, 1, 3, 256, 509, 512), 256), ((0, 130, 512), 1024), ((0, 257, 512), 4)])
def test_columns_cut_anywhere(cuts, k):
    """Buckets whose widths are no multiples of four, of a weight whose width is one."""
    sym, ctx = _weight(128, 512, k)
    b = Build(sym, ctx)
    assert b.layout([(0, 128, a, e - a) for a, e in zip(cuts, cuts[1:])], k) == _lib.MPS_OK
    assert b.emit() == _lib.MPS_OK
    np.testing.assert_array_equal(b.decoded(), sym)


def test_lists_that_are_wrong_at_first():
    """Buckets of more elements than the tensor has are refused; the right ones are accepted afterwards."""
    sym, ctx = _weight(128, 512, 5)
    b = Build(sym, ctx)
    assert b.layout([(0, 128, 0, 512), (0, 64, 0, 512)], 256) == _lib.MPS_ERR_INVALID
    assert b"more elements than the tensor" in b.lib.mps_last_error()
    assert b.layout([(0, 64, 0, 512), (64, 64, 0, 512)], 256) == _lib.MPS_OK
    assert b.emit() == _lib.MPS_OK
    np.testing.assert_array_equal(b.decoded(), sym)
