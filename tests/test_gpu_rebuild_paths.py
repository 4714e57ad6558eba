"""The rebuild and the events of the forms without lists where their paths divide: several colonies in
a handle (tile tables written by the scan's and the events' last block), one colony, and a grid of so
many bins that the scan takes a launch of its own."""
import numpy as np
import pytest

import cil_cuda_gb300 as G
from cil_cuda_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def _run(ps, sts, precision, steps, integrator, base=0):
    eng = G.Engine(ps, [4 * len(s["sigma"]) for s in sts], precision=precision, rng=G.RNG_PHILOX, seed=5,
                   integrator=integrator, rng_stream_base=base)
    for c, s in enumerate(sts):
        eng.upload(c, **s)
    out = []
    for n in steps:
        eng.step(n)
        out.append([eng.download(c) for c in range(len(ps))])
    obs = [eng.observables(c) for c in range(len(ps))]
    eng.close()
    return out, obs


@pytest.mark.parametrize("precision", [G.PREC_FP64, G.PREC_MIXED])
@pytest.mark.parametrize("integrator", [G.INTEGRATOR_EULER, G.INTEGRATOR_HEUN])
def test_batch_equals_single_colonies(gpu_lib, precision, integrator):
    # the colonies differ in size, box and rates; the same random streams alone and together
    ps, sts = [], []
    for k, n in enumerate((1, 130, 700, 40)):
        p = S.growth_params(box=25.0 + 20.0 * k, dt=1e-3, div_tau_mu=0.05 * (k + 1), div_tau_sigma=0.01, apop_rate=2.0 * k)
        ps.append(p)
        sts.append(S.disk_colony(n, p, seed=k))
    # calls of several lengths: graphs of two steps, of one step, the last step of a call
    steps = [1, 2, 31, 6]
    together, obs = _run(ps, sts, precision, steps, integrator)
    assert sum(o["ndiv_total"] for o in obs) > 50 and sum(o["napo_total"] for o in obs) > 0
    for c in range(len(ps)):
        alone, o = _run(ps[c:c + 1], sts[c:c + 1], precision, steps, integrator, base=c)
        assert o[0]["ndiv_total"] == obs[c]["ndiv_total"] and o[0]["napo_total"] == obs[c]["napo_total"]
        for a, t in zip(alone, together):
            assert a[0]["ncells"] == t[c]["ncells"]
            for k in ("sigma", "t0", "tswitch"):
                np.testing.assert_array_equal(a[0][k], t[c][k])
            if precision == G.PREC_FP64:
                np.testing.assert_array_equal(a[0]["pos"], t[c]["pos"])
            else:  # FP32 sums by shared atomics: their order is free
                d = a[0]["pos"] - t[c]["pos"]
                d -= np.round(d / ps[c]["box"][0]) * ps[c]["box"][0]
                assert np.abs(d).max() <= 1e-5


@pytest.mark.parametrize("box", [40.0, 2300.0])  # one scan block and a few; more than 4096
def test_bins_and_forces_of_small_and_huge_grids(gpu_lib, oracle_lib, box):
    p = S.base_params(2, G.FORCE_SOFTCORE, [box, box], epsilon=5.0, rcut_scale=1.0)
    st = S.disk_colony(300, p, seed=9)
    eng = G.Engine([p], [300], rng=G.RNG_DSFMT, seed=3)
    eng.upload(0, **st)
    ns, start, elems = eng.bins(0)[:3]
    width = np.asarray(box) / np.asarray(ns[:2])
    ij = np.minimum((st["pos"].reshape(-1, 2) / width).astype(np.int64), np.asarray(ns[:2]) - 1)
    key = ij[:, 0] * ns[1] + ij[:, 1]
    order = np.lexsort((np.arange(len(key)), key))
    np.testing.assert_array_equal(elems, order)
    np.testing.assert_array_equal(np.diff(start), np.bincount(key, minlength=int(ns[0]) * int(ns[1])))
    from oracle import oracle as O
    ora = O.Oracle(p, 300, 3)
    ora.set_state(**st)
    ref = ora.compute_forces()
    assert np.abs(eng.forces(0) - ref).max() <= 1e-12 * max(1.0, np.abs(ref).max())
    eng.close()


@pytest.mark.parametrize("precision,skin", [(G.PREC_FP64, 0.0), (G.PREC_MIXED, 0.0), (G.PREC_MIXED, 0.3)])
def test_captured_steps_across_uploads(gpu_lib, precision, skin):
    # states of other boxes' fill, diameters and sizes into one engine, in turn: same bin arrays (captured
    # steps go on), more bins or fewer (captured again); each leg as in an engine of its own
    p = S.growth_params(box=60.0, dt=1e-3, div_tau_mu=0.2, div_tau_sigma=0.02, apop_rate=0.5)
    states = [S.disk_colony(n, p, seed=n) for n in (300, 500, 120)]
    states.append(dict(states[0], sigma=states[0]["sigma"] * 0.5))   # twice the bins per axis
    order = [0, 0, 1, 3, 1, 2, 3, 0]

    def leg(eng, st):
        eng.upload(0, **st)
        eng.step(21)
        eng.step(8)
        return eng.download(0)

    def engine():
        return G.Engine([p], [4000], precision=precision, rng=G.RNG_PHILOX, seed=6, skin=skin)

    eng = engine()
    for k in order:
        a = leg(eng, states[k])
        fresh = engine()
        b = leg(fresh, states[k])
        fresh.close()
        assert a["ncells"] == b["ncells"]
        np.testing.assert_array_equal(a["tswitch"], b["tswitch"])
        d = a["pos"] - b["pos"]
        d -= np.round(d / 60.0) * 60.0
        assert np.abs(d).max() <= (0.0 if precision == G.PREC_FP64 else 1e-5)
    assert eng.graph_info()["graph_steps"] > 0
    eng.close()
