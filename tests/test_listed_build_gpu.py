"""The analysis that takes over the bucket lists' sort: the same histogram as without, and lists that are not those of its
scales -- another tensor's, an unwritten workspace, a wrong number of scale values -- are refused, where counters are kept per
scale and where they are not."""
import ctypes as C

import numpy as np
import pytest
import torch

from mpserve_b200 import _lib

pytestmark = pytest.mark.gpu


def _lists(lib, scales, n, ws=None):
    """(workspace, scale values) of the rows sorted by `scales`."""
    if ws is None:
        ws = torch.zeros(lib.mps_build_lists_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    buckets, values = C.c_int64(0), C.c_int64(0)
    d = torch.from_numpy(scales).cuda()
    _lib.check(lib.mps_build_lists_sort_counted(d.data_ptr(), 1, 1, 1, n, 128, ws.data_ptr(), ws.numel(), None, C.byref(buckets), C.byref(values)))
    return ws, int(values.value)


@pytest.mark.parametrize("n,m,values", [(64, 2048, 3), (64, 16, 9)])     # counters per symbol of a scale, the general form
def test_lists_of_other_scales(n, m, values):
    lib = _lib.load()
    rng = np.random.default_rng(n + m)
    ctx = torch.from_numpy(rng.integers(0, 4, (n, m)).astype(np.uint8)).cuda()
    sym = torch.from_numpy((0x3C00 + rng.integers(0, 9, (n, m))).astype(np.uint16)).cuda()
    own = (0x2000 + 5 * (np.arange(n) % values)).astype(np.uint16)
    scales = torch.from_numpy(own).cuda()
    size = lib.mps_build_workspace_bytes(n * m, n * m)
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    state = (C.c_ubyte * 256)()

    def analyze(lists, count, bytes_=None, shift=0):
        G, N = C.c_int64(-1), C.c_int64(-1)
        rc = lib.mps_build_analyze_listed(state, sym.data_ptr(), ctx.data_ptr(), scales.data_ptr(), 1, 1, 1, m, n, m, 0, 7, ws.data_ptr(), size,
                                          None if lists is None else lists.data_ptr() + shift,
                                          bytes_ if bytes_ is not None else (0 if lists is None else lists.numel()), count, None, C.byref(G), C.byref(N))
        return rc, int(G.value), int(N.value)

    want = analyze(None, 0)
    assert want[0] == _lib.MPS_OK and want[1] == 4 * values
    good, count = _lists(lib, own, n)
    assert count == values and analyze(good, count) == want
    for wrong in (count - 1, count + 1, 1, n):
        assert analyze(good, wrong)[0] == _lib.MPS_ERR_INVALID, wrong
        assert b"not those of these scales" in lib.mps_last_error()
    for wrong in (0, -1, n + 1):
        assert analyze(good, wrong)[0] == _lib.MPS_ERR_INVALID, wrong
    assert analyze(good, count, shift=2)[0] == _lib.MPS_ERR_INVALID
    assert analyze(good, count, bytes_=good.numel() - 1)[0] == _lib.MPS_ERR_WORKSPACE
    # lists of as many rows: other values, as many; the same values elsewhere; one scale; nothing written at all
    others = [own + 1, np.roll(own, 1), np.full(n, own[0]), rng.integers(0, 65536, n).astype(np.uint16)]
    for other in others:
        stale, said = _lists(lib, other.astype(np.uint16), n)
        for c in (said, count):
            assert analyze(stale, c)[0] == _lib.MPS_ERR_INVALID
    for fill in (0, 0x7F, 0xFF):
        assert analyze(torch.full_like(good, fill), count)[0] == _lib.MPS_ERR_INVALID
    assert analyze(good, count) == want      # (a refusal leaves nothing behind)
