"""A run that blows up (Lennard-Jones elements on top of each other, which move by many boxes in a step) ends
in a status or goes on, and leaves the engine whole: its bins stay within the grid."""
import numpy as np
import pytest

import cil_cuda_gb300 as G
from cil_cuda_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def _states(dim, L, n):
    p = S.base_params(dim, G.FORCE_LJ_WCA, [L] * dim, epsilon=1.0, rcut_scale=2 ** (1 / 6), noise_D=0.0)
    p["dt"] = 1e-4
    rng = np.random.default_rng(4)
    t0, tsw = S.cycle_state(rng, n, False, p["dt"])
    out = []
    for spread in (0.02, 1.0):  # on top of each other, and apart on a lattice
        side = int(np.ceil(n ** (1 / dim)))
        c = np.stack([(np.arange(n) // side ** d) % side for d in range(dim)], axis=1) * (L / side) + 0.5
        c = c if spread == 1.0 else 0.5 * L + rng.uniform(-spread, spread, (n, dim))
        pos = S.place_cells(c, S.unit_vectors(rng, n, dim), np.full(n, 0.3 if spread == 1.0 else 0.01), p["box"], p["periodic"])
        out.append(dict(pos=pos, sigma=np.full((n, 2), 0.6), t0=t0, tswitch=tsw))
    return p, out


@pytest.mark.parametrize("rng_mode", [G.RNG_PHILOX, G.RNG_DSFMT])
@pytest.mark.parametrize("precision,skin", [(G.PREC_FP64, 0.0), (G.PREC_MIXED, 0.0), (G.PREC_MIXED, 0.3)])
@pytest.mark.parametrize("dim,L,n", [(2, 2.4, 6), (2, 20.0, 40), (3, 12.0, 30)])
def test_engine_survives(gpu_lib, rng_mode, precision, skin, dim, L, n):
    p, (bad, good) = _states(dim, L, n)

    def engine():
        return G.Engine([p], [n], precision=precision, rng=rng_mode, seed=3, skin=skin)

    eng = engine()
    eng.upload(0, **bad)
    for _ in range(12):
        try:
            eng.step(3)
        except G.CilError as e:
            assert e.status in (3, 4, 5)  # capacity of a list, a force that is not finite, off the box
    g = eng.download(0, strict=False)
    d = np.abs(g["pos"] - bad["pos"])
    assert not np.isfinite(d).all() or d.max() > 0.1
    # a good state into the same engine runs as in a new one
    eng.upload(0, **good)
    eng.step(5)
    a = eng.download(0)
    eng.close()
    fresh = engine()
    fresh.upload(0, **good)
    fresh.step(5)
    b = fresh.download(0)
    fresh.close()
    assert np.abs(a["pos"] - b["pos"]).max() <= (1e-12 if precision == G.PREC_FP64 else 1e-5)
    assert np.all(np.isfinite(a["pos"]))
