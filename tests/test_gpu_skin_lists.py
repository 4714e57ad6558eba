"""The Verlet lists where their build divides: bins at the ends of periodic and open axes, boxes of a
few bins and of one, more than 64 candidates per element (past the mask), more than 1024 entries per
warp, partly filled warps, fresh elements in a handle whose capacity bounds the launch; against the
mixed form without lists, which searches the bins every step."""
import numpy as np
import pytest

import cil_cuda_gb300 as G
from cil_cuda_gb300 import synthetic as S

pytestmark = pytest.mark.gpu
# one step's displacements: FP32 pair sums in two orders, 1e-6 of a force below 2e3, times dt / zeta
TOL = 1e-6 * 2e3 * 1e-4


def _colony(dim, n, box, periodic, rcut, seed):
    p = S.base_params(dim, G.FORCE_SOFTCORE, box, epsilon=5.0, rcut_scale=rcut, noise_D=0.0)
    p["periodic"] = list(periodic) + [0] * (3 - len(periodic))
    p["dt"] = 1e-4
    rng = np.random.default_rng(seed)
    b = np.array(box[:dim])
    pos = S.place_cells(rng.uniform(0, 1, (n, dim)) * b, S.unit_vectors(rng, n, dim), np.full(n, 0.5), p["box"],
                        p["periodic"])
    for d in range(dim):
        if not p["periodic"][d]:
            pos[..., d] = np.clip(pos[..., d], 0.2, b[d] - 0.2)  # nobody leaves an open axis in the steps made
    t0, tsw = S.cycle_state(rng, n, False, p["dt"])
    return p, dict(pos=pos, sigma=rng.uniform(0.9, 1.1, (n, 2)), t0=t0, tswitch=tsw)


def _step(p, st, n, skin, steps):
    eng = G.Engine([p], [n], precision=G.PREC_MIXED, rng=G.RNG_PHILOX, seed=2, skin=skin)
    eng.upload(0, **st)
    eng.step(steps)
    g = eng.download(0)
    k = eng.skin_stats(0) if skin else None
    eng.close()
    return g["pos"], k


def _compare(p, st, n, skin=0.3, steps=2):
    a, k = _step(p, st, n, skin, steps)
    b, _ = _step(p, st, n, 0.0, steps)
    d = a - b
    for ax in range(p["dim"]):
        if p["periodic"][ax]:
            d[..., ax] -= np.round(d[..., ax] / p["box"][ax]) * p["box"][ax]
    assert np.abs(d).max() <= steps * TOL
    return k


@pytest.mark.parametrize("dim,periodic", [(2, (1, 1)), (2, (1, 0)), (2, (0, 1)), (2, (0, 0)), (3, (1, 1, 1)), (3, (1, 0, 1)),
                                          (3, (1, 1, 0))])
@pytest.mark.parametrize("bins", [2, 3, 4, 7])
def test_lists_at_the_ends_of_the_axes(gpu_lib, dim, periodic, bins):
    L = (1.1 + 0.3) * (bins + 0.2)
    n = int(0.35 * L ** dim)
    p, st = _colony(dim, n, [L] * dim, periodic, 1.0, seed=bins)
    _compare(p, st, n)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 128, 129, 1000])
def test_lists_at_warp_and_block_edges(gpu_lib, n):
    L = max(8.0, (2.2 * n) ** 0.5)
    p, st = _colony(2, n, [L, L], (1, 1), 1.0, seed=n)
    _compare(p, st, n)


@pytest.mark.parametrize("dim,rcut", [(2, 2.3), (2, 2.6), (3, 1.5)])
def test_lists_with_many_candidates(gpu_lib, dim, rcut):
    # 9 (27) bins of width rcut + skin hold well over 64 elements, the lists about 25 to 55
    n = 700 if dim == 2 else 1500
    L = (2 * n / 1.1) ** (1.0 / dim)
    p, st = _colony(dim, n, [L] * dim, (1, 1, 1)[:dim], rcut, seed=7)
    k = _compare(p, st, n)
    assert k["list_overflow"] == 0 and k["npairs"] > 10 * 2 * n  # over 1024 entries in a warp of 64 elements
    assert 2 * n / L ** dim * (3 * (1.1 * rcut + 0.3)) ** dim > 64


@pytest.mark.parametrize("cells,cap", [(1, 64), (3, 40), (200, 3000)])
def test_fresh_pairs_in_small_handles(gpu_lib, oracle_lib, cells, cap):
    # divisions between builds in handles whose capacity gives the fresh-pair kernel one block and more
    p = S.growth_params(box=25.0, dt=1e-3, div_tau_mu=0.06, div_tau_sigma=0.005, apop_rate=0.0, noise_D=0.0)
    st = S.disk_colony(cells, p, seed=3)
    res = []
    for skin in (0.3, 0.0):
        eng = G.Engine([p], [cap], precision=G.PREC_MIXED, rng=G.RNG_PHILOX, seed=4, skin=skin)
        eng.upload(0, **st)
        eng.step(90)
        res.append(eng.download(0))
        eng.close()
    a, b = res
    assert a["ncells"] == b["ncells"] > cells
    d = a["pos"] - b["pos"]
    d -= np.round(d / 25.0) * 25.0
    assert np.abs(d).max() <= 1e-4
