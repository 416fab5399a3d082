"""The tracer's passes of a warp against the walk that carries its lengths: the same bits."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# around a warp's 8 and 32 rays, a block's 16 and 64, and the change from 8 to 32 at 128 rays a multiprocessor
@pytest.mark.parametrize("count", [1, 8, 17, 33, -1, 0, 65])
@pytest.mark.parametrize("n,nz", [(1, 1), (6, 3), (16, 40)])
def test_staged_samples_equal_the_plain_walk(cuda_ok, count, n, nz):
    import torch

    from opensss_gb300 import _lib, workloads

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rays = count if count in (1, 8, 17, 33) else 128 * sms + count
    rng = np.random.default_rng(rays + n)
    size = np.ascontiguousarray(workloads.image_bounds((n, n, nz), 0.7), dtype=np.float64).reshape(-1)[:6]
    lines = rng.uniform(-1.0, 1.0, (rays, 6)) * np.abs(np.concatenate([size[3:], size[3:]])) * 2.5
    lines[::5, :2] = lines[::5, 3:5]  # along z
    lines[1::5, 2] = lines[1::5, 5]  # level
    lines[2::5] = np.round(lines[2::5] / 0.35) * 0.35  # through corners: overruns too
    lines = torch.from_numpy(lines).cuda()
    grid, cap = np.array([n, n, nz], np.int32), 2 * n + nz + 3

    def trace(lengths):
        cnt = torch.full((rays,), 77, dtype=torch.int32, device="cuda")
        idx = torch.full((rays, cap), -5, dtype=torch.int32, device="cuda")
        ln = torch.full((rays, cap), -5.0, dtype=torch.float64, device="cuda")
        sm = torch.full((rays, cap), -5.0, dtype=torch.float64, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        _lib.check(_lib.lib().sss_raytrace(
            grid.ctypes.data_as(C.c_void_p), size.ctypes.data_as(C.c_void_p), C.c_void_p(lines.data_ptr()), rays, 0, cap,
            C.c_void_p(cnt.data_ptr()), C.c_void_p(ln.data_ptr() if lengths else 0), None, C.c_void_p(idx.data_ptr()),
            C.c_void_p(sm.data_ptr()), C.c_void_p(status.data_ptr()),
            C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return cnt, idx, sm, ln, int(status.item())

    a, b = trace(True), trace(False)
    assert all(torch.equal(x.view(torch.int64) if x.dtype == torch.float64 else x,
                           y.view(torch.int64) if y.dtype == torch.float64 else y) for x, y in zip(a[:3], b[:3]))
    assert a[4] == b[4]
    # a sample is the running sum of half the lengths: they are written where the samples are
    assert torch.equal(a[3] >= 0, a[2] >= 0)
    assert torch.equal(a[2][:, 0][a[0] > 0], a[3][:, 0][a[0] > 0] / 2)
