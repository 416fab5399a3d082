"""The composed resize at the edges of its lines and taps, against the oracle and the step-by-step passes.

Tolerance as in test_gpu_prep.py: 2e-5 of the largest output value."""

import ctypes as C

import numpy as np
import pytest
import torch

from oracle import prep as P
from opensss_gb300 import _lib

pytestmark = pytest.mark.gpu
TOL = 2e-5


@pytest.mark.parametrize("shape,start,before,crop,dims", [
    ((33, 31, 32), (0, 0, 0), (0, 0, 0), (33, 31, 32), (11, 31, 33)),      # unchanged and enlarged axes
    ((40, 7, 65), (3, 0, 0), (0, 2, 0), (30, 12, 70), (7, 5, 31)),         # cut, padded both sides and behind
    ((16, 4, 5), (0, 0, 0), (0, 0, 0), (16, 4, 5), (2, 1, 1)),             # to one sample
    ((130, 9, 257), (0, 0, 0), (0, 0, 0), (130, 9, 257), (31, 20, 129)),   # lines of a multiple of 32, and one
    ((400, 4, 6), (0, 0, 0), (0, 0, 0), (400, 4, 6), (2, 4, 3)),           # more taps than the composed form holds
])
def test_composed_resize_matches_oracle_and_steps(cuda_ok, shape, start, before, crop, dims):
    from opensss_gb300.Utils import antialias_sigma

    rng = np.random.default_rng(sum(shape))
    img = (rng.gamma(2.0, 1.0, size=shape) - 0.3).astype(np.float32)
    window = np.zeros(crop, np.float64)
    src = [slice(s, min(n, s + c - b)) for s, b, c, n in zip(start, before, crop, shape)]
    part = img[tuple(src)]
    window[tuple(slice(b, b + m) for b, m in zip(before, part.shape))] = part
    ref = P.resize(window, dims)
    t = torch.from_numpy(img).cuda()
    arr = [np.array(v, np.int32) for v in (shape, start, before, crop, dims)]
    sigma = np.ascontiguousarray(antialias_sigma(arr[3], arr[4]), dtype=np.float64)
    L = _lib.lib()

    def p(a):
        return a.ctypes.data_as(C.c_void_p)

    need = int(L.sss_crop_downscale_workspace_size(p(arr[3])))
    ws = torch.empty(need + 4, dtype=torch.uint8, device="cuda")
    for shift in (0, 4):  # composed; by steps, for want of an aligned workspace
        out = torch.full(dims, np.nan, dtype=torch.float32, device="cuda")
        _lib.check(L.sss_crop_downscale(C.c_void_p(t.data_ptr()), *(p(a) for a in arr), p(sigma), 1,
                                        C.c_float(-np.inf), C.c_void_p(out.data_ptr()), C.c_void_p(ws.data_ptr() + shift),
                                        need, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        assert np.abs(out.cpu().numpy().astype(np.float64) - ref).max() <= TOL * np.abs(ref).max(), shift
