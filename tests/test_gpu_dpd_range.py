"""DPD with FP32 pair terms at the end of a pair's range, where the random force sqrt(1 - r / rc) follows
the last bits of the separation."""
import importlib.util
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def _recipe():
    spec = importlib.util.spec_from_file_location("make_dpd_golden", os.path.join(HERE, "golden", "make_dpd_golden.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


@pytest.mark.parametrize("name,dim,L", [("2d", 2, 48.0), ("3d", 3, 24.0), ("whole_axes", 2, 3.4)])
def test_pairs_at_the_end_of_their_range_keep_their_values(gpu_lib, name, dim, L):
    """The forces and velocities recorded in golden/dpd_pairs_golden.npz. A pair is alone, so its terms come
    from the same FP32 operations in the same order whatever walks the bins: equal but for an operation or
    two rounded another way after the weight (2^-23 each, under 1e-6); another rounding of the separation
    moves the random force of these pairs by 1e-4 to 1e-2 of it. The velocities add FP64 products of them
    with dt, and a position's last FP64 bit may turn an FP32 one in a pair of the three steps: 1e-5."""
    z = np.load(os.path.join(HERE, "golden", "dpd_pairs_golden.npz"))
    st = {k: z["%s.%s" % (name, k)] for k in ("pos", "sigma", "theta", "rho", "angvel", "vel")}
    got = _recipe().outputs(gpu_lib, dim, L, st)
    for k in ("ran", "dis"):
        want = z["%s.out.%s" % (name, k)]
        assert np.all(np.isfinite(want)) and np.abs(want).max() > 0
        np.testing.assert_allclose(got[k], want, rtol=1e-6, atol=1e-9 * np.abs(want).max(), err_msg=k)
    want = z["%s.out.vel" % name]
    assert np.abs(got["vel"] - want).max() <= 1e-5 * np.abs(want).max()
