"""The pair stage of several TOF bins at the edges of its chunks of 32 partners and of its rows, against the oracle."""

import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_sss import TOL, _engine, _gpu_compact, _oracle_compact, assert_same_support

pytestmark = pytest.mark.gpu


# 31, 32, 33 and 65 legs; the fewest bins, either side of 16, and a bin wider and narrower than the legs' spread
@pytest.mark.parametrize("nru,ndu", [(1, 31), (4, 8), (3, 11), (5, 13)])
@pytest.mark.parametrize("bins,width", [(2, 12.0), (16, 1.5), (17, 0.3), (33, 1.5)])
def test_histogram_pair_stage_matches_oracle(cuda_ok, att_table, nru, ndu, bins, width):
    from opensss_gb300 import workloads as W
    from opensss_gb300.batch import BatchSSS
    from opensss_gb300.engine import leg_pair_to_compact

    scanner = W.ring_scanner(4 * ndu, 2 * nru, radius_cm=20.0, ring_pitch_cm=1.0, phase=0.5)
    pr = W.make_problem(f"edge-{nru}x{ndu}-b{bins}", (12, 11, 7), 1.7, nru, ndu, bins, width, 214.0, seed=nru + bins,
                        scanner=scanner, radius_cm=8.0)
    ref = _oracle_compact(pr, att_table)
    assert np.abs(ref).max() > 0
    runs = {"plain": _gpu_compact(pr, att_table), "waves": _gpu_compact(pr, att_table, wave_points=1)}
    b = BatchSSS([(_engine(pr, att_table), pr.activity, pr.attenuation, pr.image_size)] * 2)
    for k, lp in enumerate(b.run()):
        runs[f"batch {k}"] = leg_pair_to_compact(lp.cpu().numpy(), nru, ndu)
    b.close()
    for name, got in runs.items():
        assert_same_support(got, ref)
        assert rel_l2(got, ref) < TOL, name
