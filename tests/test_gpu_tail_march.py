"""The marched tail mask against the walk of every LOR: the same bytes and status, whatever the map."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(kind, n, nz, rng):
    mu = np.zeros((n, n, nz), np.float32)
    if kind == "cylinder":
        x = np.arange(n) - (n - 1) / 2
        mu[x[:, None] ** 2 + x[None, :] ** 2 < (0.35 * n) ** 2] = 0.096
    elif kind == "sparse":  # single voxels, on the faces too
        mu = np.where(rng.random(mu.shape) < 0.01, rng.random(mu.shape), 0).astype(np.float32)
    elif kind == "dense":
        mu = rng.random(mu.shape).astype(np.float32) * 1e-3
    elif kind == "tiny":  # sums on either side of the rule's bound
        mu = np.where(rng.random(mu.shape) < 0.3, 10.0 ** rng.uniform(-12, -5, mu.shape), 0).astype(np.float32)
    elif kind == "signed":
        mu[n // 2, n // 2] = -0.01
    return mu  # "empty": all zero


@pytest.mark.parametrize("n,nz,nr,nd,af,vox", [(1, 1, 2, 40, 3, 9.0), (5, 3, 7, 64, 1, 6.0), (33, 48, 13, 126, 3, 0.9),
                                              (64, 2, 70, 40, 3, 0.6)])
@pytest.mark.parametrize("kind", ["cylinder", "sparse", "dense", "tiny", "signed", "empty"])
def test_marched_mask_equals_walked_mask(cuda_ok, kind, n, nz, nr, nd, af, vox):
    import torch

    from opensss_gb300 import DataReduction, _lib, geometry, workloads

    rng = np.random.default_rng(n + nd)
    # phase 0: lines through corners and along faces and axes; 0.37: none
    for phase, span in ((0.0, 0), (0.37, 0)) + (((0.37, 3),) if nr > 2 else ()):  # two rings have no span 3
        sc = workloads.ring_scanner(nd, nr, ring_pitch_cm=25.6 / nr, phase=phase)
        geom, pairs = sc.geometry, None
        lor, si, _ = geometry.SinogramCoordinates(1, 1, 1, 1, nd, nr, ID_Shidt=False)
        nslices = nr * nr
        if span:
            geom, _ = geometry.expandRings(sc.geometry, sc.normals)
            index = DataReduction.SinogramLUT(nr, span, nr - 1)[0]
            pairs = torch.from_numpy(DataReduction.span_ring_pairs(index).astype(np.int32)).cuda()
            nslices = pairs.shape[0]
        size = workloads.image_bounds((n, n, nz), vox)
        grid = np.array([n, n, nz], np.int32)
        bounds = np.ascontiguousarray(size, dtype=np.float64).reshape(-1)[:6]
        mu = torch.from_numpy(_map(kind, n, nz, rng).ravel(order="F")).cuda()
        g = torch.from_numpy(np.ascontiguousarray(geom, dtype=np.float64)).cuda()
        lor_d = torch.from_numpy(np.ascontiguousarray(lor, dtype=np.int16)).cuda()
        si_d = torch.from_numpy(np.ascontiguousarray(si).astype(np.int16)).cuda()
        L = _lib.lib()
        need = int(L.sss_tail_mask_workspace_size(grid.ctypes.data_as(C.c_void_p)))
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")
        for act, acf in ((0, 0.0), (1, 0.0), (0, 1.03)):
            got = []
            for nbytes in (need, need - 1, 0):  # marched, and walked for want of a workspace
                out = torch.zeros(((nd + 1) * (nd // 2), nslices), dtype=torch.uint8, device="cuda")
                status = torch.zeros(1, dtype=torch.int32, device="cuda")
                _lib.check(L.sss_tail_mask_marched(
                    grid.ctypes.data_as(C.c_void_p), bounds.ctypes.data_as(C.c_void_p), C.c_void_p(mu.data_ptr()), act,
                    geom.shape[0], nd, C.c_void_p(g.data_ptr()), C.c_void_p(lor_d.data_ptr()),
                    C.c_void_p(si_d.data_ptr()), C.c_void_p(pairs.data_ptr() if span else 0),
                    nslices if span else 0, nslices, af, acf, C.c_void_p(out.data_ptr()),
                    C.c_void_p(status.data_ptr()), C.c_void_p(ws.data_ptr() if nbytes else 0), nbytes,
                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
                got.append((out, int(status.item())))
            for out, status in got[1:]:
                assert torch.equal(out, got[0][0]) and status == got[0][1]
