"""The FP64 force pass against the oracle at the edges of its work split: lanes per element (chosen
from the colony's size), blocks and warps that are partly filled, bins at the ends of the axes
(periodic images, open axes), more survivors per element than one batch holds."""
import numpy as np
import pytest

import cil_cuda_gb300 as G
from cil_cuda_gb300 import synthetic as S

pytestmark = pytest.mark.gpu

# FP64 sums of at most a few hundred terms: reordering and a few units of the last place per term
TOL = 1e-12


def _state(p, n, seed, sigma=1.0, spread=0.1):
    rng = np.random.default_rng(seed)
    D = p["dim"]
    box = np.array(p["box"][:D])
    centres = rng.uniform(0, 1, (n, D)) * box
    ax = S.unit_vectors(rng, n, D)
    pos = S.place_cells(centres, ax, np.full(n, 0.5 * sigma), p["box"], p["periodic"])
    for d in range(D):
        if not p["periodic"][d]:
            pos[..., d] = np.clip(pos[..., d], 0.0, np.nextafter(box[d], 0.0))
    sig = sigma * rng.uniform(1 - spread, 1 + spread, (n, 2))
    t0, tsw = S.cycle_state(rng, n, False, p["dt"])
    return dict(pos=pos, sigma=sig, t0=t0, tswitch=tsw)


def _check(p, st, n):
    from oracle import oracle as O
    eng = G.Engine([p], [n], rng=G.RNG_DSFMT, seed=3)
    eng.upload(0, **st)
    got = eng.forces(0)
    ora = O.Oracle(p, n, 3)
    ora.set_state(**st)
    ref = ora.compute_forces()
    eng.close()
    assert np.abs(got - ref).max() <= TOL * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("law", [G.FORCE_SOFTCORE, G.FORCE_HERTZ, G.FORCE_LJ_WCA])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 1217, 4864, 4865, 9729, 19457])
def test_forces_at_lane_and_block_edges(dim, law, n):
    L = max(4.2, (1.7 * n) ** (1.0 / dim))
    p = S.base_params(dim, law, [L] * dim, epsilon=5.0, rcut_scale=2 ** (1 / 6) if law == G.FORCE_LJ_WCA else 1.0)
    _check(p, _state(p, n, seed=n), n)


@pytest.mark.parametrize("dim,periodic", [(2, (1, 0)), (2, (0, 1)), (2, (0, 0)), (3, (1, 1, 0)), (3, (0, 1, 1))])
@pytest.mark.parametrize("bins", [3, 4, 7])
def test_forces_at_the_ends_of_the_axes(dim, periodic, bins):
    # boxes of a few bins, open and periodic axes: every image and clipped row is met
    p = S.base_params(dim, G.FORCE_SOFTCORE, [1.2 * bins] * dim, epsilon=5.0, rcut_scale=1.0)
    p["periodic"] = list(periodic) + [0] * (3 - dim)
    n = 40 * bins if dim == 2 else 60 * bins
    _check(p, _state(p, n, seed=bins), n)


@pytest.mark.parametrize("n", [400, 6000, 30000])
def test_forces_with_many_contacts(n):
    # about 60 contacts per element: several batches of survivors at every lane count
    L = (n * 2 / 20.0) ** 0.5
    p = S.base_params(2, G.FORCE_SOFTCORE, [L, L], epsilon=1.0, rcut_scale=1.0)
    _check(p, _state(p, n, seed=n, sigma=1.0), n)


@pytest.mark.parametrize("scale", [1e-6, 1e4])
def test_forces_far_from_unit_lengths(scale):
    # the FP32 range test follows the box and the coordinates, whatever their unit
    n = 900
    L = 40.0 * scale
    p = S.base_params(2, G.FORCE_SOFTCORE, [L, L], epsilon=5.0, rcut_scale=1.0, kappa=0.0, motility=[0.0, 0.0],
                      noise_D=0.0)
    p["periodic"] = [1, 0, 0]
    _check(p, _state(p, n, seed=5, sigma=scale), n)
