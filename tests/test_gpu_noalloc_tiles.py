"""cil_bin_elements_noalloc at the edges of its radix tiles, warps and scan blocks, one and two radix
passes, clustered elements; against a stable sort of the bin keys on the host (whole numbers, equal),
and on a stream of the caller's, captured and replayed with other positions."""
import numpy as np
import pytest

import cil_cuda_gb300 as G

pytestmark = pytest.mark.gpu


def _expected(pos, box, ns):
    dim = pos.shape[1]
    key = np.zeros(len(pos), np.int64)
    for d in range(dim):
        v = (pos[:, d] * (1.0 / box[d]) * float(ns[d])).astype(np.int64)
        key = key * ns[d] + np.clip(v, 0, ns[d] - 1)
    nb = int(np.prod(ns[:dim]))
    start = np.concatenate([[0], np.cumsum(np.bincount(key, minlength=nb))])
    return start, np.argsort(key, kind="stable")


def _call(torch, pos, box, width, max_bins, stream=None):
    n, dim = pos.shape
    ns = np.zeros(3, np.int32)
    start = torch.full((max_bins + 1,), -1, dtype=torch.int32, device="cuda")
    elems = torch.full((max(n, 1),), -1, dtype=torch.int32, device="cuda")
    st = G.lib().cil_bin_elements_noalloc(pos.data_ptr(), n, dim, G._dp(box), width, G._ip(ns), start.data_ptr(),
                                          elems.data_ptr(), max_bins, stream)
    assert st == 0
    return ns, start, elems


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 31, 33, 255, 256, 257, 2047, 2048, 2049, 4097, 100003, 1 << 20])
@pytest.mark.parametrize("bins", [2, 900, 1100, 60000])
def test_tile_edges(gpu_lib, n, dim, bins):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + bins)
    side = bins ** (1.0 / dim)
    box = np.array([side * 1.5 + 0.2] * dim)
    pos = rng.random((n, dim)) * box
    if n > 300:
        pos[n // 3: n // 2] = pos[0]  # a sixth of the elements in one bin
    p = torch.from_numpy(pos).cuda()
    ns, start, elems = _call(torch, p, box, 1.5, 1 << 20)
    want_start, want = _expected(pos, box, ns)
    nb = len(want_start) - 1
    np.testing.assert_array_equal(start.cpu().numpy()[:nb + 1], want_start)
    np.testing.assert_array_equal(elems.cpu().numpy()[:n], want)


@pytest.mark.parametrize("L,width", [(1.0, 0.001), (1254.3, 1.31), (3e-5, 1e-6), (7.7e5, 1.0), (100.0, 1.0)])
def test_positions_next_to_the_bins_edges(gpu_lib, L, width):
    # one FP64 step to either side of an edge, and parts of an FP32 step: where the FP32 product cannot
    # tell the bin
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(8)
    box = np.array([L, 40.0 * width])
    n = 20000
    ns0 = int(L / (width + min(box) * 1e-8))
    x = rng.integers(0, ns0, n) * (L / ns0)
    x *= 1.0 + rng.choice([0.0, 1e-16, -1e-16, 3e-16, -3e-16, 1e-12, -1e-12, 1e-8, -1e-8, 1e-7, -1e-7, 1e-6, -1e-6], n)
    x[:4] = [0.0, 5e-324, 1e-40, np.nextafter(L, 0.0)]
    pos = np.stack([np.clip(x, 0.0, np.nextafter(L, 0.0)), rng.random(n) * box[1]], axis=1)
    p = torch.from_numpy(pos).cuda()
    ns, start, elems = _call(torch, p, box, width, 1 << 20) if ns0 * 39 <= 1 << 20 else (None, None, None)
    if ns is None:  # too many bins along with the other axis: one wide axis less
        box = np.array([L, 3.2 * width])
        pos[:, 1] = rng.random(n) * box[1]
        p = torch.from_numpy(pos).cuda()
        if ns0 * 3 > 1 << 20:
            width *= 4.0
            box[1] = 3.2 * width
            pos[:, 1] = rng.random(n) * box[1]
            p = torch.from_numpy(pos).cuda()
        ns, start, elems = _call(torch, p, box, width, 1 << 20)
    want_start, want = _expected(pos, box, ns)
    np.testing.assert_array_equal(start.cpu().numpy()[:len(want_start)], want_start)
    np.testing.assert_array_equal(elems.cpu().numpy()[:n], want)


def test_captured_on_a_stream_of_the_callers(gpu_lib):
    torch = pytest.importorskip("torch")
    n, box = 5000, np.array([120.0, 120.0])
    rng = np.random.default_rng(3)
    pos = [rng.random((n, 2)) * box for _ in range(2)]
    p = torch.from_numpy(pos[0]).cuda()
    _call(torch, p, box, 1.5, 1 << 14)  # the device's first call comes before any capture
    torch.cuda.synchronize()
    ns = np.zeros(3, np.int32)
    start = torch.zeros((1 << 14) + 1, dtype=torch.int32, device="cuda")
    elems = torch.zeros(n, dtype=torch.int32, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        p.mul_(1.0)  # a kernel of the caller's before the call, and one after
        st = G.lib().cil_bin_elements_noalloc(p.data_ptr(), n, 2, G._dp(box), 1.5, G._ip(ns), start.data_ptr(),
                                              elems.data_ptr(), 1 << 14, torch.cuda.current_stream().cuda_stream)
        twice = elems * 2
    assert st == 0
    for q in pos:
        p.copy_(torch.from_numpy(q))
        g.replay()
        torch.cuda.synchronize()
        want_start, want = _expected(q, box, ns)
        np.testing.assert_array_equal(start.cpu().numpy()[:len(want_start)], want_start)
        np.testing.assert_array_equal(elems.cpu().numpy(), want)
        np.testing.assert_array_equal(twice.cpu().numpy(), 2 * want)
