"""The histogram by tiles against the two-pass form: the same prompts, randoms and normalisation."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _records(n, words, rng, ncr, nr, tof):
    ev = rng.integers(0, 2**32, (n, words), dtype=np.uint64).astype(np.uint32)
    ev[:, 0] >>= rng.integers(0, 31, n).astype(np.uint32)  # event[0]: any number of bits, 0 too
    ev[:, -3] = tof.astype(np.float32).view(np.uint32)
    ev[:, -2:] = rng.integers(0, ncr * nr, (n, 2))
    return ev


# events around a block's 1024; bins from one to the most that 32 cells of a tile hold
@pytest.mark.parametrize("n", [0, 1, 1023, 1025, 40000])
@pytest.mark.parametrize("bins,mash,values", [(1, 1, True), (6, 2, True), (13, 1, False), (575, 2, True), (576, 2, False)])
def test_tiles_equal_the_two_pass_form(cuda_ok, n, bins, mash, values):
    import torch

    from opensss_gb300 import Datafile, _lib, geometry

    rng = np.random.default_rng(n + bins)
    nd, nr, words, duration = 40, 5, 6, 597.3 if mash == 1 else 75.0 * bins
    lor, si, _ = geometry.SinogramCoordinates(1, 1, 1, 1, nd, nr, ID_Shidt=False)
    lor, si = np.asarray(lor).astype(np.int16), np.asarray(si).astype(np.int16)
    # TOF on, beside and between the bin edges, outside the range and not a number
    edges = (np.arange(n) % (bins + 1)) * (2000.0 / bins) - 1000.0
    tof = np.where(np.arange(n) % 3 == 0, edges, np.where(np.arange(n) % 3 == 1, edges * (1 + 1e-7),
                                                          rng.uniform(-1100, 1100, n)))
    tof[5::97], tof[6::97], tof[7::97] = np.nan, np.inf, -np.inf
    ev = torch.from_numpy(_records(n, words, rng, nd * mash, nr, tof).view(np.uint8).reshape(-1)).cuda()
    if n == 40000:  # one cell far beyond 65535 events in sum with the tiles' other cells
        ev = ev.reshape(n, -1)
        ev[: n // 2, 4 * (words - 2):] = ev[0, 4 * (words - 2):]
        ev = ev.reshape(-1).repeat(4)
    lor_t, si_t = torch.from_numpy(lor).cuda(), torch.from_numpy(si).cuda()
    shape = (int(lor[:, :, 1].max()) + 1, int(lor[:, :, 0].max()) + 1, int(si.max()) + 1)
    M = Datafile.sino_map(lor_t, nd, mash, 0, si_t, *shape, bins, 1000.0)
    L = _lib.ListmodeLayout(4 * words, 4 * (words - 2), 4 * (words - 3), 4 * (words - 3))
    n = ev.numel() // (4 * words)
    lib = _lib.lib()

    def ptr(t):
        return C.c_void_p(0 if t is None else t.data_ptr())

    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    status = torch.zeros(2, dtype=torch.int32, device="cuda")
    counts = torch.zeros((*shape, bins), dtype=torch.int32, device="cuda")
    last = torch.zeros(shape, dtype=torch.int64, device="cuda") if values else None
    want = [torch.full((*shape, bins), -1, dtype=torch.int16, device="cuda"),
            torch.zeros(shape, device="cuda") if values else None, torch.ones(shape, device="cuda") if values else None]
    _lib.check(lib.sss_histogram_prompts(ptr(ev), n, C.byref(L), C.byref(M), ptr(counts), ptr(last), ptr(status), st))
    _lib.check(lib.sss_histogram_finish(ptr(ev), n, C.byref(L), C.byref(M), ptr(counts), ptr(last), duration,
                                        *(ptr(t) for t in want), st))
    need = int(lib.sss_histogram_tiled_workspace_size(n, C.byref(M), int(values)))
    assert need > 0
    ws = torch.full((need,), 255, dtype=torch.uint8, device="cuda")
    got = [None if t is None else torch.full_like(t, -7) for t in want]
    _lib.check(lib.sss_histogram_tiled(ptr(ev), n, C.byref(L), C.byref(M), duration, *(ptr(t) for t in got), ptr(ws), need,
                                       ptr(status[1:]), st))
    for a, b in zip(got, want):
        assert a is None or torch.equal(a.view(torch.int32) if a.dtype == torch.float32 else a,
                                        b.view(torch.int32) if b.dtype == torch.float32 else b)
    assert int(status[0]) == int(status[1])
    # FP64 restatement of the bins and of the randoms values
    e = ev.cpu().numpy().view(np.uint32).reshape(n, words)
    if values and n:
        used = want[1].cpu().numpy()
        x = ((e[:, 0].astype(np.float64) * duration) / bins).astype(np.float32)
        assert np.isin(used[used != 0], x).all()
    M.tof_bins = 1 << 20  # a cell's counters beyond a tile: the two-pass form's
    assert lib.sss_histogram_tiled_workspace_size(n, C.byref(M), int(values)) == 0
