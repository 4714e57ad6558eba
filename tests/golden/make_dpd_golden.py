"""Recipe of dpd_pairs_golden.npz: DPD with FP32 pair terms (precision 1) near the end of a pair's range.

The random force takes sqrt(w), w = 1 - r / rc, in FP32, so for a pair at the end of its range its last
bits follow from how the separation was rounded. The file keeps what the library gave on a GB300 when the
dissipative and random forces had a kernel of their own over records relative to the bins' origins: the
forces after the upload and the velocities after three steps.

    python tests/golden/make_dpd_golden.py OUT.npz    (from the root of a built tree)
"""
import os
import sys

import numpy as np

sys.path.insert(0, os.getcwd())
SIG0 = 1.1283791670955126


def pairs(rng, dim, L, spacing, count):
    """Pairs of cells around grid points (the first ones across the periodic boundary), 3e-6 to 1e-3 of
    their range inside it. A pair's range is the diameter of the cell of lower index."""
    per = int(round(L / spacing))
    at = np.array([[(k // per ** d) % per for d in range(dim)] for k in range(count)]) * spacing
    u = rng.normal(size=(count, dim))
    u /= np.linalg.norm(u, axis=1)[:, None]
    sigma = SIG0 * rng.uniform(0.95, 1.05, 2 * count)
    r = sigma[0::2] * (1 - 10.0 ** rng.uniform(-5.5, -3.0, count))
    pos = np.empty((2 * count, dim))
    pos[0::2] = at - 0.4 * r[:, None] * u
    pos[1::2] = at + 0.6 * r[:, None] * u
    return np.mod(pos, L), sigma


def cases():
    rng = np.random.default_rng(2024)
    for name, dim, L, spacing, count in (("2d", 2, 48.0, 4.0, 128), ("3d", 3, 24.0, 4.0, 128), ("whole_axes", 2, 3.4, 3.4, 1)):
        pos, sigma = pairs(rng, dim, L, spacing, count)
        n = len(sigma)
        yield name, dim, L, dict(pos=pos, sigma=sigma, theta=rng.uniform(0, 0.5, n), rho=np.ones(n),
                                 angvel=np.full(n, 1e-4), vel=rng.normal(0, 0.05, (n, dim)))


def params(G, dim, L):
    return dict(dim=dim, box=[L] * dim + [0.0] * (3 - dim), periodic=[1, 1, 1], dt=1e-4, motility=1.0, v1=15.0,
                integrator=G.CYCLE_DPD, mass=1.0, kbt=0.003, dis_diff=1.0, dis_bg=0.01, precision=1)


def outputs(G, dim, L, st):
    eng = G.CycleEngine(params(G, dim, L), 2 * len(st["sigma"]) + 8, seed=17)
    eng.upload(**st)
    first = eng.download()
    eng.step(3)
    last = eng.download()
    eng.close()
    return dict(ran=first["force_ran"], dis=first["force_dis"], con=first["force"], vel=last["vel"])


if __name__ == "__main__":
    import cil_cuda_gb300 as G
    keep = {}
    for name, dim, L, st in cases():
        keep.update({"%s.%s" % (name, k): v for k, v in st.items()})
        keep.update({"%s.out.%s" % (name, k): v for k, v in outputs(G, dim, L, st).items()})
    np.savez_compressed(sys.argv[1], **keep)
