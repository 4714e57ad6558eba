"""A colony uploaded again into a skin-mode engine: the scheduler's statistics restart with the new
state, so the divisions and apoptoses of the earlier run (whose totals go on counting) are not taken
for events of the new run's first step."""
import pytest

import cil_cuda_gb300 as G
from cil_cuda_gb300 import skin_scheduler
from cil_cuda_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("colonies", [1, 3])
def test_scheduler_statistics_restart_with_the_upload(gpu_lib, colonies):
    p = S.growth_params(box=60.0, dt=1e-3, div_tau_mu=0.1, div_tau_sigma=0.01, apop_rate=1.0)
    st = S.disk_colony(300, p, seed=4)
    eng = G.Engine([p] * colonies, [2000] * colonies, precision=G.PREC_MIXED, rng=G.RNG_PHILOX, seed=2,
                   skin=skin_scheduler.load()[2])
    skin_scheduler.install(eng)
    for c in range(colonies):
        eng.upload(c, **st)
    eng.step(1)
    first = [eng.sched_state(c) for c in range(colonies)]
    eng.step(80)
    for c in range(colonies):
        ob = eng.observables(c)
        assert ob["ndiv_total"] > 20 and ob["napo_total"] > 0
        eng.upload(c, **st)
    eng.step(1)  # the rates are taken before this step's events
    for c in range(colonies):
        q, f = eng.sched_state(c), first[c]
        assert q["div_rate"] == f["div_rate"] == 0.0 and q["apo_rate"] == f["apo_rate"] == 0.0
        # 3, 4: displacements of the last step; 5, 6: event rates; 10: trips of the guard
        for k in (0, 3, 4, 5, 6):
            assert q["features"][k] == f["features"][k], k
        assert eng.observables(c)["ndiv_total"] > 20  # the totals go on counting
    eng.close()
