"""Thousands of cells that divide in the same step (a colony of one age): the queue of due cells is filled in
no order, and beyond 2048 of them their order comes from a scan of the colony's cells."""
import time

import numpy as np
import pytest

import cil_cuda_gb300 as G
from cil_cuda_gb300 import synthetic as S

pytestmark = pytest.mark.gpu
FORMS = [(G.PREC_FP64, 0.0), (G.PREC_MIXED, 0.0), (G.PREC_MIXED, 0.3)]
NEVER = 2**30


def _colony(n, box, share, seed=1):
    p = S.growth_params(box=box, dt=1e-5, div_tau_mu=100.0, div_tau_sigma=1.0, apop_rate=0.0, noise_D=0.0)
    st = S.disk_colony(n, p, seed=seed, phi=0.3)
    rng = np.random.default_rng(seed)
    due = np.sort(rng.choice(n, int(share * n), replace=False))
    st["t0"] = np.zeros(n, np.int32)
    st["tswitch"] = np.full(n, NEVER, np.int32)
    st["tswitch"][due] = 4
    return p, st, due


@pytest.mark.parametrize("precision,skin", FORMS)
@pytest.mark.parametrize("n,share", [(600, 1.0), (2049, 1.0), (3000, 0.69), (9000, 0.7), (9000, 0.2)])
def test_daughters_come_in_cell_order(gpu_lib, precision, skin, n, share):
    p, st, due = _colony(n, 400.0, share)
    eng = G.Engine([p, p], [2 * n + 8, 64], precision=precision, rng=G.RNG_PHILOX, seed=3, skin=skin)
    eng.upload(0, **st)
    eng.upload(1, **_colony(20, 400.0, 0.5, seed=2)[1])
    eng.step(6)
    g, other = eng.download(0), eng.download(1)
    eng.close()
    assert g["ncells"] == n + len(due) and other["ncells"] == 30
    # the k-th due cell's daughter is cell n + k, at its mother's place
    d = g["pos"][n:].mean(axis=1) - g["pos"][due].mean(axis=1)
    assert np.abs(d - np.round(d / 400.0) * 400.0).max() < 2.0
    first = st["pos"][due].mean(axis=1) - g["pos"][due].mean(axis=1)
    assert np.abs(first - np.round(first / 400.0) * 400.0).max() < 2.0
    rest = np.setdiff1d(np.arange(n), due)
    assert np.all(g["tswitch"][rest] == NEVER) and np.all(g["t0"][n:] == 4) and np.all(g["t0"][due] == 4)


@pytest.mark.parametrize("precision,skin", FORMS)
def test_a_step_of_many_divisions_stays_short(gpu_lib, precision, skin):
    # 80 000 at once: a sort of the queue by one block took 15 to 17 ms
    n = 80000
    p, st, _ = _colony(n, 1200.0, 1.0)
    eng = G.Engine([p], [2 * n + 8], precision=precision, rng=G.RNG_PHILOX, seed=3, skin=skin)
    best = 1e9
    for _ in range(3):
        eng.upload(0, **st)
        eng.step(2)
        t0 = time.perf_counter()
        eng.step(3)
        best = min(best, time.perf_counter() - t0)
        assert eng.download(0)["ncells"] == 2 * n
    eng.close()
    assert best < 9e-3
