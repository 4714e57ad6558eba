"""The cell-cycle model's pair kernels against the restatement where their work split changes: blocks
and warps that are partly filled, the lanes per cell (from the colony's size), bins at the ends of
periodic and open axes and axes of one or two bins, more pairs in range than a warp's batch holds."""
import numpy as np
import pytest

import cil_cuda_gb300 as G

pytestmark = pytest.mark.gpu
SIG0 = 1.1283791670955126
# forces and pressures are FP64 sums of a few hundred terms at most, each within a few units of the
# last place except a contact length A = sqrt of a difference, whose rounding 1e-16 ra^2 / A stays
# below 1e-12 for every overlap a draw of 1e5 pairs meets (h > 1e-8); three steps of dt / zeta 1e-3
TOL = 1e-10


def _state(n, box, dim, seed, spread=0.2):
    rng = np.random.default_rng(seed)
    return dict(pos=rng.uniform(0, 1, (n, dim)) * np.asarray(box[:dim]),
                sigma=SIG0 * rng.uniform(1 - spread, 1 + spread, n), theta=rng.uniform(0, 0.9, n),
                rho=rng.uniform(0.5, 1.0, n), angvel=np.full(n, 2e-3), vel=rng.normal(0, 0.2, (n, dim)))


def _check(prm, st, n, steps=3):
    from oracle import oracle as O
    cap = n + 8
    eng = G.CycleEngine(prm, cap, seed=11)
    eng.upload(**st)
    eng.step(steps)
    g = eng.download()
    eng.close()
    o = O.CycleOracle(prm, cap, 11)
    o.set_state(**st)
    assert o.step(steps) == 0
    s = o.state()
    assert g["ncells"] == s["ncells"] == n
    for k in ("pos", "vel", "force", "force_dis", "force_ran", "pressure", "sigma", "sigma_t", "theta", "rho"):
        a, b = np.asarray(g[k]), np.asarray(s[k])
        d = a - b
        if k == "pos":
            L = np.asarray(prm["box"][:d.shape[1]])
            d = d - np.where(np.asarray(prm["periodic"][:d.shape[1]]) > 0, np.round(d / L) * L, 0.0)
        assert np.abs(d).max() <= TOL * max(1.0, np.abs(b).max()), k


def _params(dim, box, integrator, periodic=(1, 1, 1)):
    p = dict(dim=dim, box=box, periodic=list(periodic), dt=2e-4, motility=1.0, zeta=0.2, v1=15.0)
    if integrator == G.CYCLE_DPD:
        p.update(integrator=integrator, mass=1.0, kbt=0.01, dis_diff=2.0, dis_bg=0.5)
    return p


@pytest.mark.parametrize("integrator", [0, G.CYCLE_DPD])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 129, 2000, 4864, 4865, 9729, 19457])
def test_lane_and_block_edges(gpu_lib, oracle_lib, n, dim, integrator):
    L = max(4.0, (1.5 * n) ** (1.0 / dim))
    box = [L, L, L]
    _check(_params(dim, box, integrator), _state(n, box, dim, seed=n), n)


@pytest.mark.parametrize("dim,periodic", [(2, (1, 0, 0)), (2, (0, 1, 0)), (2, (0, 0, 0)), (3, (1, 1, 0)), (3, (0, 1, 1))])
@pytest.mark.parametrize("bins", [1.5, 2.2, 3.1, 4.4, 7.0])
def test_ends_of_the_axes(gpu_lib, oracle_lib, dim, periodic, bins):
    L = 1.05 * 1.2 * SIG0 * bins
    box = [L, L, L]
    n = int(6 * bins ** dim)
    for integrator in (0, G.CYCLE_DPD):
        st = _state(n, box, dim, seed=int(10 * bins))
        st["pos"] = 0.1 * L + 0.8 * st["pos"] * 1.0  # open axes: nobody leaves within the steps
        _check(_params(dim, box, integrator, periodic), st, n)


@pytest.mark.parametrize("n", [300, 6000, 30000])
def test_many_pairs_in_range(gpu_lib, oracle_lib, n):
    # about 25 cells within reach of each: several batches at every lane count
    L = (n / 25.0) ** 0.5
    box = [L, L, 0.0]
    prm = _params(2, box, 0)
    prm["zeta"] = 2000.0  # deep overlaps: the cells hardly move in the steps compared
    _check(prm, _state(n, box, 2, seed=n, spread=0.05), n)


@pytest.mark.parametrize("growth", [1.2, 2.5])
def test_cells_that_outgrow_their_bins_within_a_call(gpu_lib, oracle_lib, growth):
    # targets far above the diameters: the search widens by itself (5 and more bins across)
    n, box = 400, [30.0, 30.0, 0.0]
    prm = _params(2, box, 0)
    prm.update(v1=15.0 * growth * 40, divide=1)
    st = _state(n, box, 2, seed=5)
    st["theta"][:] = 0.0
    st["angvel"][:] = 1e-6
    _check(prm, st, n, steps=30)


@pytest.mark.parametrize("integrator", [0, G.CYCLE_DPD])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 33, 600, 1023, 1024, 1025, 3000])
def test_many_cells_divide_at_once(gpu_lib, oracle_lib, n, dim, integrator):
    # every cell reaches phase 1 in the same step (queue and scan of k_cy_divide, daughters in mother
    # order), then half of the colony's capacity is used
    from oracle import oracle as O
    L = max(6.0, (3.0 * n) ** (1.0 / dim))
    box = [L, L, L]
    prm = _params(dim, box, integrator)
    st = _state(n, box, dim, seed=n)
    st["theta"] = np.full(n, 0.999)
    st["rho"] = np.ones(n)
    eng = G.CycleEngine(prm, 2 * n, seed=7)
    eng.upload(**st)
    eng.step(1)
    g = eng.download()
    eng.close()
    o = O.CycleOracle(prm, 2 * n, 7)
    o.set_state(**st)
    assert o.step(1) == 0
    s = o.state()
    assert g["ncells"] == s["ncells"] == 2 * n
    for k in ("pos", "sigma", "sigma_t", "theta", "rho", "angvel", "vel"):
        d = np.asarray(g[k]) - np.asarray(s[k])
        if k == "pos":
            d -= np.round(d / L) * L
        assert np.abs(d).max() <= TOL * max(1.0, np.abs(s[k]).max()), k


@pytest.mark.parametrize("integrator", [0, G.CYCLE_DPD])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 1000])
def test_state_comes_back_as_uploaded(gpu_lib, n, dim, integrator):
    L = max(6.0, (3.0 * n) ** (1.0 / dim))
    box = [L, L + 1.0, L + 2.0]
    st = _state(n, box, dim, seed=n)
    eng = G.CycleEngine(_params(dim, box, integrator), n + 5, seed=1)
    keys = ("pos", "vel", "sigma", "theta", "rho", "angvel")
    for _ in range(2):
        eng.upload(**st)
        g = eng.download()
        assert g["ncells"] == n
        for k in keys:
            np.testing.assert_array_equal(g[k], st[k])
        st["pos"] = st["pos"][::-1].copy()
    eng.upload(**st)
    for d in range(dim):  # refused, and the state stays
        bad = dict(st, pos=st["pos"].copy(), sigma=2 * st["sigma"])
        bad["pos"][n // 2, d] = box[d]
        with pytest.raises(G.CilError) as e:
            eng.upload(**bad)
        assert e.value.status == 5
        g = eng.download()
        for k in keys:
            np.testing.assert_array_equal(g[k], st[k])
    eng.close()
