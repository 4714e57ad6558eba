"""The mixed form without lists repeats itself bit for bit: an element's pairs are summed in slot order and
the slots follow the bins and the element ids, whatever else is in the handle and whether the steps are
launched or replayed from a capture made for another state."""
import numpy as np
import pytest

import cil_cuda_gb300 as G
from cil_cuda_gb300 import synthetic as S

pytestmark = pytest.mark.gpu
KEYS = ("pos", "vel", "sigma", "t0", "tswitch")


def _engine(ps, caps, integrator, base=0, graphs=True):
    return G.Engine(ps, caps, precision=G.PREC_MIXED, rng=G.RNG_PHILOX, seed=5, integrator=integrator,
                    rng_stream_base=base, graphs=graphs)


def _same(a, b):
    assert a["ncells"] == b["ncells"]
    for k in KEYS:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("integrator", [G.INTEGRATOR_EULER, G.INTEGRATOR_HEUN])
def test_batch_single_and_launched(gpu_lib, integrator):
    ps, sts = [], []
    for k, n in enumerate((1, 130, 700, 40)):
        ps.append(S.growth_params(box=25.0 + 20.0 * k, dt=1e-3, div_tau_mu=0.05 * (k + 1), div_tau_sigma=0.01,
                                  apop_rate=2.0 * k))
        sts.append(S.disk_colony(n, ps[-1], seed=k))

    def legs(which, base, graphs):
        eng = _engine([ps[c] for c in which], [4 * len(sts[c]["sigma"]) for c in which], integrator, base, graphs)
        for i, c in enumerate(which):
            eng.upload(i, **sts[c])
        out = []
        for n in (1, 2, 31, 6):
            eng.step(n)
            out.append([eng.download(i) for i in range(len(which))])
        eng.close()
        return out

    together = legs(range(4), 0, True)
    for other in (legs(range(4), 0, True), legs(range(4), 0, False)):
        for a, b in zip(together, other):
            for c in range(4):
                _same(a[c], b[c])
    for c in range(4):
        for a, b in zip(together, legs([c], c, True)):
            _same(a[c], b[0])


def test_captured_steps_across_uploads(gpu_lib):
    p = S.growth_params(box=60.0, dt=1e-3, div_tau_mu=0.2, div_tau_sigma=0.02, apop_rate=0.5)
    states = [S.disk_colony(n, p, seed=n) for n in (300, 500, 120)]
    states.append(dict(states[0], sigma=states[0]["sigma"] * 0.5))  # twice the bins per axis

    def leg(eng, st):
        eng.upload(0, **st)
        eng.step(21)
        eng.step(8)
        return eng.download(0)

    eng = _engine([p], [4000], G.INTEGRATOR_EULER)
    for k in (0, 0, 1, 3, 1, 2, 3, 0):
        fresh = _engine([p], [4000], G.INTEGRATOR_EULER)
        _same(leg(eng, states[k]), leg(fresh, states[k]))
        fresh.close()
    eng.close()


def test_many_cells_twice(gpu_lib):
    p = S.growth_params(box=700.0, dt=1e-3, div_tau_mu=0.05, div_tau_sigma=0.005, apop_rate=0.5)
    st = S.disk_colony(100000, p, seed=4)
    out = []
    for _ in range(2):
        eng = _engine([p], [250000], G.INTEGRATOR_EULER)
        eng.upload(0, **st)
        eng.step(40)
        out.append(eng.download(0))
        eng.close()
    assert out[0]["ncells"] > 120000
    _same(*out)
