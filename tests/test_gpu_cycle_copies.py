"""The cell-cycle model's copies into ordinary (pageable) host arrays."""
import time

import numpy as np
import pytest

import cil_cuda_gb300 as G

pytestmark = pytest.mark.gpu


def _engine(n, integrator):
    side = int(np.ceil(np.sqrt(n)))
    rng = np.random.default_rng(2)
    pos = np.stack([np.arange(n) % side, np.arange(n) // side], axis=1) * 1.15 + 0.5 + rng.uniform(-0.02, 0.02, (n, 2))
    p = dict(box=[1.15 * side + 2.0] * 2 + [0.0], dt=1e-5, motility=1.0, zeta=0.2, v1=15.0)
    if integrator == G.CYCLE_DPD:
        p.update(integrator=integrator, mass=1.0, kbt=0.003, dis_diff=1.0, dis_bg=0.01, precision=1)
    eng = G.CycleEngine(p, n + 100, seed=7)
    eng.upload(pos=pos, theta=rng.uniform(0, 0.5, n), rho=np.ones(n), angvel=np.full(n, 1e-5))
    return eng


@pytest.mark.parametrize("integrator", [0, G.CYCLE_DPD])
@pytest.mark.parametrize("n", [100, 8191, 8193, 50000])  # vectors below and above 64 KB
def test_downloads_repeat_themselves(gpu_lib, integrator, n):
    eng = _engine(n, integrator)
    eng.step(2)
    a, b = eng.download(), eng.download()
    eng.close()
    assert a["ncells"] == n
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    assert np.all(a["sigma"] > 0) and np.all(np.isfinite(a["force"])) and np.abs(a["vel"]).max() > 0


@pytest.mark.parametrize("integrator", [0, G.CYCLE_DPD])
def test_a_download_into_new_arrays_stays_short(gpu_lib, integrator):
    # 0.6M cells into arrays that nobody has touched: 51 and 59 ms when the copies faulted their pages in
    eng = _engine(600000, integrator)
    t = []
    for _ in range(5):
        t0 = time.perf_counter()
        eng.download()
        t.append(time.perf_counter() - t0)
    eng.close()
    assert min(t) < 15e-3
