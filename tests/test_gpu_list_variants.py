"""Which form of the list force kernel runs: the one asked for, or with none asked for the library's
choice by the number of cells."""
import re

import pytest

import cil_cuda_gb300 as G
from cil_cuda_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def _form(n, **kw):
    """(chunks in flight, blocks an SM, cells per block) of the k_force_cells instance that a step launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda").add_(1)
    p = S.growth_params(box=1024.0, dt=1e-4, divide=0, apop_rate=0.0)
    eng = G.Engine([p], [n + 8], precision=G.PREC_MIXED, rng=G.RNG_PHILOX, seed=4, skin=0.3, **kw)
    eng.upload(0, **S.disk_colony(n, p, seed=2))
    eng.step(2)
    for _ in range(2):  # the first profile of a process may miss its launches
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            torch.zeros(1, device="cuda").add_(1)
            eng.step(2)
            torch.cuda.synchronize()
        names = {e.name for e in prof.events() if "k_force_cells" in e.name}
        if names:
            break
    eng.close()
    if not names:
        pytest.skip("the profiler saw no kernels here")
    (name,) = names
    _, _, chunks, blocks, cells = re.search(r"k_force_cells<(\d+), (\d+), (\d+), (\d+), (\d+)", name).groups()
    return int(chunks), int(blocks), int(cells)


@pytest.mark.parametrize("n", [2000, 120000])
@pytest.mark.parametrize("staging,occupancy", [(4, 3), (4, 0), (0, 3), (2, 3), (1, 3), (1, 4)])
def test_the_form_asked_for_runs(gpu_lib, n, staging, occupancy):
    assert _form(n, staging=staging, occupancy=occupancy) == (staging or 4, 2 * (occupancy or 3), 128)


@pytest.mark.parametrize("block", [256, 512])
def test_other_block_sizes_keep_their_form(gpu_lib, block):
    assert _form(120000, block_size=block) == (4, {256: 3, 512: 1}[block], block)


def test_the_default_follows_the_cells(gpu_lib):
    # 6 blocks of 128 cells on each of 152 SMs hold 116 736
    assert _form(2000) == (4, 6, 128)
    assert _form(120000) == (4, 8, 128)
