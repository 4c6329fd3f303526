"""Shared-table decode with chunk lists that are not in the builder's order: the table of a chunk is the one of the
stream that lists it, chunks that no stream lists are not decoded, and the form with scratch answers like the form
without."""
import ctypes as C

import numpy as np
import pytest
import torch

from mpserve_b200 import _lib
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

KEYS = ("bitstream_u64", "decode_syms_i16", "decode_nbits_u8", "scale_bit_base_i64", "chunk_startbit_rel_u32", "chunk_out_base_u32",
        "chunk_meta_u32", "chunk_scale_id_i32", "out_idx_i32", "stream_chunk_ofs_i64", "stream_chunk_ids_i32")


def _decode(art, out_len, scratch, L=11):
    lib = _lib.load()
    d = {key: torch.from_numpy(np.ascontiguousarray(art[key])).cuda() for key in KEYS}
    out = torch.full((out_len,), 0x1234, dtype=torch.int16, device="cuda")
    S, NC = d["decode_syms_i16"].size(0), d["chunk_meta_u32"].numel()
    args = [d["bitstream_u64"].data_ptr(), d["bitstream_u64"].numel(), d["decode_syms_i16"].data_ptr(), d["decode_nbits_u8"].data_ptr(), S,
            d["scale_bit_base_i64"].data_ptr(), d["scale_bit_base_i64"].numel(), d["chunk_startbit_rel_u32"].data_ptr(),
            d["chunk_out_base_u32"].data_ptr(), d["chunk_meta_u32"].data_ptr(), d["chunk_scale_id_i32"].data_ptr(), NC,
            d["out_idx_i32"].data_ptr(), d["stream_chunk_ofs_i64"].data_ptr(), d["stream_chunk_ids_i32"].data_ptr(), out_len, L,
            out.data_ptr()]
    stream = torch.cuda.current_stream().cuda_stream
    if scratch:
        ws = torch.empty(lib.mps_shared_workspace_bytes(S, NC), dtype=torch.uint8, device="cuda")
        _lib.check(lib.mps_decode_awq_shared_table_ws(*args, ws.data_ptr(), ws.numel(), stream))
    else:
        _lib.check(lib.mps_decode_awq_shared_table(*args, stream))
    torch.cuda.synchronize()
    return out.cpu().numpy().view(np.uint16)


def _weight(n, m, runs, seed, scales):
    rng = np.random.default_rng(seed)
    ctx = np.repeat(rng.integers(0, 16, (n, (m + runs - 1) // runs)), runs, axis=1)[:, :m].astype(np.uint8)
    sym = (0x3C00 + rng.integers(0, 500, (n, m))).astype(np.uint16)
    sc = (0x3C00 + np.arange(n) % scales).astype(np.uint16)
    return sym, ctx, sc


@pytest.mark.parametrize("n,m,runs,scales", [(1, 1, 1, 1), (1, 1023, 1, 1), (5, 1025, 3, 2), (64, 2048, 1, 40), (3, 4096, 700, 3),
                                             (4200, 16, 1, 4200)])     # the last: more streams than 16 bits hold
@pytest.mark.parametrize("order", ["built", "reversed", "partial"])
def test_both_forms_follow_the_lists(n, m, runs, scales, order):
    sym, ctx, sc = _weight(n, m, runs, n + m, scales)
    L = 8 if scales > 4000 else 11
    art = dict(orc.build_awq_shared(sym, ctx, sc, L))
    ofs, ids = art["stream_chunk_ofs_i64"].copy(), art["stream_chunk_ids_i32"].copy()
    want = sym.reshape(-1).copy()
    if order == "reversed":                       # any order within a stream
        for s in np.flatnonzero(np.diff(ofs) > 1):
            ids[ofs[s]:ofs[s + 1]] = ids[ofs[s]:ofs[s + 1]][::-1].copy()
    elif order == "partial" and ids.size > 4:     # the last streams' chunks are listed by nobody
        kept = int(ofs[np.searchsorted(ofs, ids.size // 2)])
        ofs = np.minimum(ofs, kept)
        base, meta = art["chunk_out_base_u32"], art["chunk_meta_u32"] >> 8
        for c in ids[kept:]:
            want[base[c]:base[c] + meta[c]] = 0x1234
    art["stream_chunk_ofs_i64"], art["stream_chunk_ids_i32"] = ofs, ids
    np.testing.assert_array_equal(_decode(art, n * m, False, L), want)
    np.testing.assert_array_equal(_decode(art, n * m, True, L), want)


def test_a_chunk_is_decoded_with_the_table_of_the_stream_that_lists_it():
    sym, ctx, sc = _weight(4, 512, 1, 9, 1)
    art = dict(orc.build_awq_shared(sym, ctx, sc, 11))
    ofs = art["stream_chunk_ofs_i64"].copy()
    ofs[1:-1] = np.maximum(ofs[1:-1] - 3, 0)      # the first three chunks of every stream change hands
    art["stream_chunk_ofs_i64"] = np.maximum.accumulate(ofs)
    got = _decode(art, sym.size, True)
    np.testing.assert_array_equal(got, _decode(art, sym.size, False))
    assert not np.array_equal(got, sym.reshape(-1))


def test_scratch_is_checked():
    assert _lib.load().mps_shared_workspace_bytes(16, 0) == 0
    assert _lib.load().mps_shared_workspace_bytes(0xFFFE, 10) == 20 and _lib.load().mps_shared_workspace_bytes(0xFFFF, 10) == 40
    sym, ctx, sc = _weight(1, 64, 1, 3, 1)
    art = dict(orc.build_awq_shared(sym, ctx, sc, 11))
    d = {key: torch.from_numpy(np.ascontiguousarray(art[key])).cuda() for key in KEYS}
    p = C.c_void_p(d["bitstream_u64"].data_ptr())
    rc = _lib.load().mps_decode_awq_shared_table_ws(p, 1, p, p, 16, p, 2, p, p, p, p, 5, p, p, p, 64, 11, p, p, 4, None)
    assert rc == _lib.MPS_ERR_WORKSPACE


class _Calls:
    """The library, with the names of the functions that are called."""

    def __init__(self, lib):
        self.lib, self.names = lib, []

    def __getattr__(self, name):
        self.names.append(name)
        return getattr(self.lib, name)


@pytest.mark.parametrize("over", [-1, 0, 1])
def test_few_chunks_take_one_launch(over, monkeypatch):
    """Scratch, with its two launches more, from a number of chunks on at which it pays; the same values on both sides."""
    import MPServe_cuda
    from mpserve_b200 import api

    sym, ctx, sc = _weight(16, 640, 1, 3, 5)
    art = dict(orc.build_awq_shared(sym, ctx, sc, 11))
    chunks = art["chunk_meta_u32"].size
    assert chunks < api.SHARED_ONE_KERNEL_CHUNKS <= 1 << 20
    if over >= 0:
        monkeypatch.setattr(api, "SHARED_ONE_KERNEL_CHUNKS", chunks - over)
    calls = _Calls(_lib.load())
    monkeypatch.setattr(api._lib, "load", lambda: calls)
    d = {key: torch.from_numpy(np.ascontiguousarray(art[key])).cuda() for key in KEYS}
    got = MPServe_cuda.huffman_decode_awq_shared_table(*[d[key] for key in KEYS], sym.size, 11)
    assert ("mps_decode_awq_shared_table_ws" in calls.names) == (over == 1)
    np.testing.assert_array_equal(got.cpu().numpy().view(np.uint16), sym.reshape(-1))


@pytest.mark.parametrize("scales,L,values", [(2, 8, 900), (40, 8, 900), (3, 11, 9000), (2047, 6, 70), (2048, 6, 70), (1, 3, 40)])
@pytest.mark.parametrize("misaligned", [False, True])
def test_escape_codes_among_single_symbols(scales, L, values, misaligned):
    """Tables with ESC entries beside tables without, in streams of which a block of positions meets one and many, on both
    sides of the number that leaves a mark its bit; code lengths at an address that is no multiple of 16."""
    rng = np.random.default_rng(scales + L)
    n, m = max(scales, 24), 256
    ctx = rng.integers(0, 16, (n, m)).astype(np.uint8)
    sym = (0x3C00 + np.where(ctx < 3, rng.integers(0, values, (n, m)), rng.integers(0, min(1 << L, 9), (n, m)))).astype(np.uint16)
    sc = (0x3C00 + np.arange(n) % scales).astype(np.uint16)
    art = dict(orc.build_awq_shared(sym, ctx, sc, L))
    if misaligned:
        keep = torch.zeros(art["decode_nbits_u8"].size + 16, dtype=torch.uint8, device="cuda")
        view = keep[3:3 + art["decode_nbits_u8"].size].view(art["decode_nbits_u8"].shape)
        view.copy_(torch.from_numpy(np.ascontiguousarray(art["decode_nbits_u8"])))
        lib = _lib.load()
        d = {key: torch.from_numpy(np.ascontiguousarray(art[key])).cuda() for key in KEYS}
        d["decode_nbits_u8"] = view
        S, NC = d["decode_syms_i16"].size(0), d["chunk_meta_u32"].numel()
        out = torch.zeros(n * m, dtype=torch.int16, device="cuda")
        ws = torch.empty(lib.mps_shared_workspace_bytes(S, NC), dtype=torch.uint8, device="cuda")
        _lib.check(lib.mps_decode_awq_shared_table_ws(
            d["bitstream_u64"].data_ptr(), d["bitstream_u64"].numel(), d["decode_syms_i16"].data_ptr(), view.data_ptr(), S,
            d["scale_bit_base_i64"].data_ptr(), d["scale_bit_base_i64"].numel(), d["chunk_startbit_rel_u32"].data_ptr(),
            d["chunk_out_base_u32"].data_ptr(), d["chunk_meta_u32"].data_ptr(), d["chunk_scale_id_i32"].data_ptr(), NC,
            d["out_idx_i32"].data_ptr(), d["stream_chunk_ofs_i64"].data_ptr(), d["stream_chunk_ids_i32"].data_ptr(), n * m, L,
            out.data_ptr(), ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream))
        got = out.cpu().numpy().view(np.uint16)
    else:
        got = _decode(art, n * m, True, L)
    np.testing.assert_array_equal(got, _decode(art, n * m, False, L))
    np.testing.assert_array_equal(got, orc.decode_awq_shared(art, n * m, L).reshape(-1).view(np.uint16))
