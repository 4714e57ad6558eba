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


@pytest.mark.parametrize("dim", [2, 3])
def test_pairs_within_a_few_units_of_their_range(gpu_lib, dim):
    """r below rc by 0 to 3 units of 2^-24: the FP32 quotient r / rc rounds past 1 for some per cent of the pairs
    whose r2 is the number below rc^2 (diameters between 0.9 and 1 have most), and the weight under the root is 0 then, not negative. sqrt(w) is at
    most sqrt(2^-19) (the units, and the FP32 rounding of coordinates below 2 with their differences), a
    normal from 24-bit uniforms at most 5.77."""
    m, L, count = _recipe(), 400.0 if dim == 2 else 88.0, 10000
    rng = np.random.default_rng(5 + dim)
    pos, sigma = m.pairs(rng, dim, L, 4.0, count)
    sigma *= 0.86
    u = pos[1::2] - pos[0::2]
    u -= np.round(u / L) * L
    u /= np.linalg.norm(u, axis=1)[:, None]
    pos[1::2] = np.mod(pos[0::2] + sigma[0::2, None] * (1 - rng.integers(0, 4, count) * 2.0**-24)[:, None] * u, L)
    n = len(sigma)
    st = dict(pos=pos, sigma=sigma, theta=np.zeros(n), rho=np.ones(n), angvel=np.full(n, 1e-4),
              vel=np.full((n, dim), 0.05))
    p = m.params(gpu_lib, dim, L)
    eng = gpu_lib.CycleEngine(p, n, seed=3)
    eng.upload(**st)
    ran = eng.download()["force_ran"]
    eng.step(2)
    eng.close()
    assert np.all(np.isfinite(ran)) and np.count_nonzero(ran) > n // 8
    assert np.abs(ran).max() <= np.sqrt(2 * p["dis_diff"] * p["kbt"]) * np.sqrt(2.0**-19) * 5.77
