"""Which streams of the shared-table layout are marked as perhaps having ESC codes: none at table sizes where a mark costs more
than it saves; beyond, those whose tables hold one and those whose tables are too many or too large to be looked at for a stretch
of the index.  The marks lie in the scratch after a call."""
import numpy as np
import pytest
import torch

from mpserve_b200 import _lib
from oracle import oracle as orc
from tests.test_shared_order_gpu import KEYS

pytestmark = pytest.mark.gpu

POSITIONS, TABLES, LOOK_BYTES, MIN_LEN = 2048, 8, 65536, 9


@pytest.mark.parametrize("scales,L,wide", [(1, 8, 0), (1, 9, 0), (40, 9, 0), (1, 11, 0), (3, 11, 0), (2, 14, 0), (9, 14, 0), (1, 15, 0), (4, 15, 0),
                                           (1, 14, 16), (1, 14, 17), (30, 11, 12)])
def test_marks(scales, L, wide):
    """`wide`: the tables spread to that many bits, as a caller's own encoder may make them."""
    rng = np.random.default_rng(scales * 32 + L)
    n, m = 240, 256
    ctx = rng.integers(0, 16, (n, m)).astype(np.uint8)
    sym = (0x3C00 + ctx.astype(np.int64) * 16 + rng.integers(0, 9, (n, m))).astype(np.uint16)
    esc = (1 << min(L, 11)) + 60                     # context 5 of the first scale sees more symbols than a short table has slots
    here = (ctx == 5) & (np.arange(n) % scales == 0)[:, None]
    sym[here] = 0x3C00 + np.arange(here.sum()) % esc
    sc = (0x3C00 + np.arange(n) % scales).astype(np.uint16)
    art = dict(orc.build_awq_shared(sym, ctx, sc, L))
    for key in ("decode_syms_i16", "decode_nbits_u8"):
        art[key] = np.repeat(art[key], 1 << max(wide - L, 0), axis=1)
    L = max(wide, L)
    d = {key: torch.from_numpy(np.ascontiguousarray(art[key])).cuda() for key in KEYS}
    S, chunks = art["decode_syms_i16"].shape[0], art["chunk_meta_u32"].size
    lib = _lib.load()
    out = torch.zeros(n * m, dtype=torch.int16, device="cuda")
    ws = torch.empty(lib.mps_shared_workspace_bytes(S, chunks), dtype=torch.uint8, device="cuda")
    _lib.check(lib.mps_decode_awq_shared_table_ws(
        d["bitstream_u64"].data_ptr(), d["bitstream_u64"].numel(), d["decode_syms_i16"].data_ptr(), d["decode_nbits_u8"].data_ptr(), S,
        d["scale_bit_base_i64"].data_ptr(), d["scale_bit_base_i64"].numel(), d["chunk_startbit_rel_u32"].data_ptr(),
        d["chunk_out_base_u32"].data_ptr(), d["chunk_meta_u32"].data_ptr(), d["chunk_scale_id_i32"].data_ptr(), chunks,
        d["out_idx_i32"].data_ptr(), d["stream_chunk_ofs_i64"].data_ptr(), d["stream_chunk_ids_i32"].data_ptr(), n * m, L,
        out.data_ptr(), ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream))
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint16), sym.reshape(-1))
    owner = ws.cpu().numpy().view(np.uint16)
    ofs, ids = art["stream_chunk_ofs_i64"], art["stream_chunk_ids_i32"]
    holds = (art["decode_nbits_u8"] & 0x80).any(axis=1)
    stream = np.searchsorted(ofs, np.arange(ids.size), side="right") - 1
    want = np.zeros(ids.size, bool)
    for p in range(0, ids.size, POSITIONS):
        met = stream[p:p + POSITIONS]
        streams = met[-1] - met[0] + 1
        looked = streams <= TABLES and streams << L <= LOOK_BYTES
        want[p:p + POSITIONS] = holds[met] if looked else True
    if L < MIN_LEN:
        want[:] = False
    np.testing.assert_array_equal(owner[ids] & 0x7FFF, stream)
    np.testing.assert_array_equal((owner[ids] >> 15).astype(bool), want)
