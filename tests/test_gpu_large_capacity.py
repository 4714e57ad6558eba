"""Engines whose capacity is far above their cells: an early colony in an engine sized for its end. The
force passes' grids follow the cells known of, the results do not depend on them, and a step takes about
what it takes in a small engine."""
import time

import numpy as np
import pytest

import cil_cuda_gb300 as G
from cil_cuda_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def _early(n=500, dim=2):
    p = S.growth_params(box=256.0, dt=1e-4, divide=0, apop_rate=0.0, noise_D=0.0)
    return p, S.disk_colony(n, p, seed=3)


def _engine(p, cap, precision, skin):
    return G.Engine([p], [cap], precision=precision, rng=G.RNG_PHILOX, seed=4, skin=skin)


@pytest.mark.parametrize("precision", [G.PREC_FP64, G.PREC_MIXED])
def test_results_do_not_depend_on_the_capacity(gpu_lib, precision):
    # FP64: 8 lanes per element, then 2 and 1. Without lists every sum has its order: equal. (With lists their
    # order is that of the cells' arrival in the bins, which differs from run to run.)
    p, st = _early()
    got = []
    for cap in (600, 200000, 300000):
        eng = _engine(p, cap, precision, 0.0)
        eng.upload(0, **st)
        eng.step(20)
        got.append(eng.download(0))
        eng.close()
    for g in got[1:]:
        np.testing.assert_array_equal(g["pos"], got[0]["pos"])


def test_growth_past_the_grid_within_one_call(gpu_lib):
    """131 000 cells in lists (1024 tiles of 128, 2048 blocks) that grow past 262 144 (2048 tiles) within
    one call, so that blocks take several tiles, against calls of 20 steps, whose grids follow. dt 1e-5: a
    step's displacements agree to 1e-6 of a force below 2e3 (FP32 sums in two orders, as fresh pairs
    arrive by atomics), and a tile left out would leave stale positions behind."""
    p = S.growth_params(box=1500.0, dt=1e-5, div_tau_mu=1.2e-3, div_tau_sigma=5e-5, apop_rate=0.0, noise_D=0.0)
    st = S.disk_colony(131000, p, seed=5, phi=0.15)
    steps, got = 240, []
    for call in (steps, 20):
        eng = _engine(p, 700000, G.PREC_MIXED, 0.3)
        eng.upload(0, **st)
        for _ in range(steps // call):
            eng.step(call)
        got.append(eng.download(0))
        eng.close()
    a, b = got
    assert a["ncells"] == b["ncells"] > 300000
    np.testing.assert_array_equal(a["tswitch"], b["tswitch"])
    d = a["pos"] - b["pos"]
    d -= np.round(d / 1500.0) * 1500.0
    assert np.abs(d).max() <= steps * 1e-6 * 2e3 * 1e-5


@pytest.mark.parametrize("precision,skin,cap,most", [(G.PREC_FP64, 0.0, 1000000, 2.0), (G.PREC_MIXED, 0.3, 2000000, 1.4)])
def test_a_step_costs_about_as_much_in_a_large_engine(gpu_lib, precision, skin, cap, most):
    # blocks for every tile and lane of the capacity: 5 times (FP64) and 1.65 times the small engine's
    p, st = _early()
    best = []
    for c in (600, cap):
        eng = _engine(p, c, precision, skin)
        eng.upload(0, **st)
        eng.step(40)
        t = []
        for _ in range(25):
            t0 = time.perf_counter()
            eng.step(40)
            t.append(time.perf_counter() - t0)
        best.append(min(t))
        eng.close()
    assert best[1] <= most * best[0]


def _dilute(box, n=3000):
    p = S.growth_params(box=box, dt=1e-4, divide=0, apop_rate=0.0, noise_D=0.0)
    return p, S.disk_colony(n, p, seed=6)


def test_lists_over_more_bins_than_scan_blocks(gpu_lib):
    """13.6M bins, whose 13 300 scan blocks are taken in turn by 4096: two steps in lists against the bins
    of every step (FP32 pair sums in two orders, 1e-6 of a force below 2e3, times dt / zeta)."""
    p, st = _dilute(6000.0)
    pos = []
    for skin in (0.3, 0.0):
        eng = _engine(p, 3000, G.PREC_MIXED, skin)
        eng.upload(0, **st)
        eng.step(2)
        pos.append(eng.download(0)["pos"])
        eng.close()
    assert np.abs(pos[0] - pos[1]).max() <= 2 * 1e-6 * 2e3 * 1e-4


def test_lists_cost_about_as_much_over_many_bins(gpu_lib):
    # a step that rebuilds nothing passes the scan kernels by: a block per scan block took 1.9 times
    best = []
    for box in (1500.0, 6000.0):
        p, st = _dilute(box)
        eng = _engine(p, 3000, G.PREC_MIXED, 0.3)
        eng.upload(0, **st)
        eng.step(40)
        t = []
        for _ in range(25):
            t0 = time.perf_counter()
            eng.step(40)
            t.append(time.perf_counter() - t0)
        best.append(min(t))
        eng.close()
    assert best[1] <= 1.5 * best[0]
