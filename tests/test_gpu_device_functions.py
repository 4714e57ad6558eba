"""Device functions by themselves: a probe compiled from csrc's headers, with and without FMA contraction
(the library's translation units use both)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from cil_cuda_gb300 import build as B

pytestmark = pytest.mark.gpu

PROBE = r"""
#include "cil_internal.cuh"
using namespace cil;

template <int LAW>
__global__ void k_reaches(ColonyConst C, int n, const float4 *p, const float2 *u, float si, float skin, int *in) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float ui[2] = {u[i].x, u[i].y};
  in[i] = list_reaches<2, LAW>(C, ui, si, skin, p[i], 1, 0) ? 1 : 0;
}

template <class T>
static T *up(const void *src, size_t bytes) {
  void *q = nullptr;
  if (cudaMalloc(&q, bytes) != cudaSuccess) return nullptr;
  cudaMemcpy(q, src, bytes, cudaMemcpyHostToDevice);
  return static_cast<T *>(q);
}

__global__ void k_moved(ColonyConst C, int n, const float *u, const int *h, int *bin, int *shift) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) bin[i] = moved_bin(C, 0, h[i], u[i], shift + i);
}

extern "C" int moved(int periodic, int ns, float bw, int n, const float *u, const int *h, int *bin, int *shift) {
  ColonyConst C{};
  C.ns[0] = ns;
  C.periodic[0] = periodic;
  C.bwf[0] = bw;
  C.inv_bwf[0] = 1.0f / bw;
  float *du = up<float>(u, 4 * size_t(n));
  int *dh = up<int>(h, 4 * size_t(n)), *db = up<int>(bin, 4 * size_t(n)), *ds = up<int>(shift, 4 * size_t(n));
  k_moved<<<(n + 127) / 128, 128>>>(C, n, du, dh, db, ds);
  cudaMemcpy(bin, db, 4 * size_t(n), cudaMemcpyDeviceToHost);
  const cudaError_t e = cudaMemcpy(shift, ds, 4 * size_t(n), cudaMemcpyDeviceToHost);
  cudaFree(du);
  cudaFree(dh);
  cudaFree(db);
  cudaFree(ds);
  return static_cast<int>(e);
}

// rsqrt_pos, sqrt_from, rcp_normal, CUDA's rsqrt, sqrt and reciprocal, the two approximate seeds, mid_range
__global__ void k_roots(int n, const double *a, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i], y = rsqrt_pos(x);
  double s, r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(s) : "d"(x));
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double v[9] = {y, sqrt_from(x, y), rcp_normal(x), rsqrt(x), sqrt(x), 1.0 / x, s, r, mid_range(x) ? 1.0 : 0.0};
  for (int k = 0; k < 9; ++k) out[size_t(k) * n + i] = v[k];
}

extern "C" int roots(int n, const double *a, double *out) {
  double *da = up<double>(a, 8 * size_t(n)), *dout = up<double>(out, 72 * size_t(n));
  k_roots<<<(n + 127) / 128, 128>>>(n, da, dout);
  const cudaError_t e = cudaMemcpy(out, dout, 72 * size_t(n), cudaMemcpyDeviceToHost);
  cudaFree(da);
  cudaFree(dout);
  return static_cast<int>(e);
}

extern "C" int reaches(int well, int n, const float *p, const float *u, float si, float skin, float rcs, float xi,
                       int *in) {
  ColonyConst C{};
  C.rcs_f = rcs;
  C.well_sigma_f = xi;
  C.bwf[0] = C.bwf[1] = 2.0f;
  float4 *dp = up<float4>(p, 16 * size_t(n));
  float2 *du = up<float2>(u, 8 * size_t(n));
  int *di = up<int>(in, 4 * size_t(n));
  if (well)
    k_reaches<CIL_FORCE_SC><<<(n + 127) / 128, 128>>>(C, n, dp, du, si, skin, di);
  else
    k_reaches<CIL_FORCE_SOFTCORE><<<(n + 127) / 128, 128>>>(C, n, dp, du, si, skin, di);
  const cudaError_t e = cudaMemcpy(in, di, 4 * size_t(n), cudaMemcpyDeviceToHost);
  cudaFree(dp);
  cudaFree(du);
  cudaFree(di);
  return static_cast<int>(e);
}
"""


@pytest.fixture(scope="module")
def probes(tmp_path_factory):
    d = tmp_path_factory.mktemp("probe")
    src = d / "probe.cu"
    src.write_text(PROBE)
    out, running = {}, []
    for fmad in ("true", "false"):
        so = str(d / ("probe_%s.so" % fmad))
        running.append((fmad, so, subprocess.Popen([B.nvcc(), *B.ARCH, "-O3", "-std=c++17", "--fmad=" + fmad, "-shared",
                                                    "-Xcompiler", "-fPIC", "-I", os.path.join(B.ROOT, "include"),
                                                    "-I", B.CSRC, str(src), "-o", so])))
    for fmad, so, p in running:
        assert p.wait() == 0
        out[fmad] = C.CDLL(so)
    return out


def _fma32(a, b, c):
    # products and sums of FP32 numbers within a few binades of each other are exact in 64 bits
    return (a.astype(np.float64) * b + c).astype(np.float32)


@pytest.mark.parametrize("well", [0, 1])
def test_list_reach_rounds_as_stated(gpu_lib, probes, well):
    """The list build decides each pair in two kernels, which must agree in the last bit: the sums and
    products of the decision are the stated ones, whatever the compiler may contract. Pairs within a
    unit of the last place of the reach, where a sum of rounded squares decides some the other way."""
    rng = np.random.default_rng(8)
    f = np.float32
    si, sj, skin, rcs, xi = f(1.0371), f(0.9713), f(0.31), f(1.0923), f(0.0517)
    sij = f(0.5) * (si + sj)
    if well:
        sij = sij + xi
    cut = _fma32(np.array([rcs]), np.array([sij]), skin)[0]
    n = 200000
    d = np.empty((n, 2), f)
    d[:, 0] = rng.uniform(0.1, 0.9, n) * cut
    d[:, 1] = np.sqrt(np.float64(cut) ** 2 - d[:, 0].astype(np.float64) ** 2)
    u = np.zeros((n, 2), f)  # the element at its bin's origin: the differences are the records' own
    p = np.zeros((n, 4), f)
    p[:, :2] = d
    p[:, 3] = -sj  # a record with its sign set counts by its magnitude
    want = _fma32(d[:, 1], d[:, 1], d[:, 0] * d[:, 0]) < cut * cut
    other = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] < cut * cut
    assert 0 < want.sum() < n and (want != other).sum() > n // 100
    for lib in probes.values():
        got = np.zeros(n, np.int32)
        a = [np.ascontiguousarray(v) for v in (p, u)]
        assert lib.reaches(well, n, a[0].ctypes.data_as(C.c_void_p), a[1].ctypes.data_as(C.c_void_p), C.c_float(si),
                           C.c_float(skin), C.c_float(rcs), C.c_float(xi), got.ctypes.data_as(C.c_void_p)) == 0
        np.testing.assert_array_equal(got.astype(bool), want)


def _roots(lib, a):
    a = np.ascontiguousarray(a, np.float64)
    out = np.empty((9, len(a)))
    assert lib.roots(len(a), a.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p)) == 0
    return out


def _mid_range_values():
    """Random mantissas at every exponent of mid_range (2^-511 to 2^510), and both ends of each binade."""
    rng = np.random.default_rng(12)
    e = np.arange(-511, 510)
    one = np.ldexp(1.0, e)
    ends = np.concatenate([one * (1 + k * 2.0**-52) for k in range(4)] + [one * (2 - k * 2.0**-52) for k in range(1, 5)])
    m = 1 + rng.integers(0, 2**52, 600000) * 2.0**-52
    # the operand's low 32 bits, which the seeds ignore, all 0 and all 1
    top = 1 + rng.integers(0, 2**20, 100000) * 2.0**-20
    m = np.concatenate([m, top, top + 2.0**-20 - 2.0**-52])
    return np.concatenate([ends, np.ldexp(m, rng.integers(-511, 510, len(m)))])


def test_roots_and_reciprocals_within_their_bounds(gpu_lib, probes):
    """The FP64 kernels' reciprocal square root, root and reciprocal against the values (in longer
    arithmetic) and CUDA's results over mid_range. Seeds good to 2^-19 leave series terms below 2^-55 and
    2^-57. rsqrt_pos: the last sum's rounding 2^-53, half of e's 2^-53 and the series 0.16 x 2^-53: 1.75 x
    2^-53. sqrt_from: the last rounding, and terms below 2^-100: 0.501 units. rcp_normal: 1.1 x 2^-53. CUDA's
    sqrt and division are correctly rounded and its rsqrt within a unit: at most 1, 1 and 2 units apart."""
    a = _mid_range_values()
    x = a.astype(np.longdouble)
    assert np.finfo(np.longdouble).nmant >= 63
    for lib in probes.values():
        rs, sq, rc, c_rs, c_sq, c_rc, seed_rs, seed_rc, mid = _roots(lib, a)
        assert np.all(mid == 1.0)
        root = np.sqrt(x)
        assert np.abs(seed_rs * root - 1).max() <= 2.0**-19
        assert np.abs(seed_rc * x - 1).max() <= 2.0**-19
        assert np.abs(rs * root - 1).max() <= 1.75 * 2.0**-53
        assert (np.abs(sq - root) / np.spacing(sq)).max() <= 0.501
        assert np.abs(rc * x - 1).max() <= 1.1 * 2.0**-53
        for got, cuda, units in ((rs, c_rs, 2), (sq, c_sq, 1), (rc, c_rc, 1)):
            assert (np.abs(got - cuda) / np.spacing(cuda)).max() <= units


def test_mid_range_takes_its_range_only(gpu_lib, probes):
    tiny, big = 2.0**-511, 2.0**510
    out = [0.0, -0.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, tiny * (1 - 2.0**-53), big, 1e300, 1e-300]
    ins = [tiny, 1.0, big * (1 - 2.0**-53)]
    for lib in probes.values():
        mid = _roots(lib, np.array(out + ins))[8]
        assert list(mid) == [0.0] * len(out) + [1.0] * len(ins)


@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("ns", [1, 3, 40])
def test_a_moved_bin_is_in_the_grid(gpu_lib, probes, periodic, ns):
    """Whatever an element's FP32 coordinate has become (an unstable run), its bin is one of the grid's;
    within a grid's length of a periodic axis it is the wrapped one, along an open one the clamped one."""
    rng = np.random.default_rng(3)
    bw = np.float32(1.5)  # quotients of multiples of 3/4 are exact enough for their floors
    near = 0.75 * rng.integers(-2 * ns, 2 * ns + 1, 4000) + 0.3
    far = np.concatenate([s * 10.0 ** rng.uniform(0, 38, 2000) for s in (-1, 1)])
    u = np.concatenate([near, far, [np.inf, -np.inf, np.nan, 0.0, -0.0, 3e38, -3e38]]).astype(np.float32)
    h = rng.integers(0, ns, len(u)).astype(np.int32)
    for lib in probes.values():
        b, sh = np.full(len(u), -7, np.int32), np.zeros(len(u), np.int32)
        p = [x.ctypes.data_as(C.c_void_p) for x in (u, h, b, sh)]
        assert lib.moved(periodic, ns, C.c_float(bw), len(u), *p) == 0
        assert b.min() >= 0 and b.max() < ns
        want = h[:4000] + np.floor(u[:4000] / bw).astype(np.int64)
        if periodic:
            inside = (want >= -ns) & (want < 2 * ns)
            np.testing.assert_array_equal(b[:4000][inside], (want % ns)[inside])
            np.testing.assert_array_equal(sh[:4000], want - h[:4000])
        else:
            np.testing.assert_array_equal(b[:4000], np.clip(want, 0, ns - 1))
            np.testing.assert_array_equal(sh[:4000], b[:4000] - h[:4000])
