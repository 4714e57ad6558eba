// cil_bin_elements_noalloc: element binning (the counting sort of cil_bins) for callers
// that cannot allocate device memory.
//
// Who needs it: applications that hand this library only memory they already own — a host
// framework with its own budgeted device pool that forbids outside cudaMalloc, or a real-time
// loop that cannot afford an allocation's latency or its failure mid-run. The caller passes
// device input and output buffers; the scratch (bin keys, the radix pass's packed ids, bin
// counts, per-tile digit histograms, scan partials) lives in file-scope __device__ arrays
// below, so nothing is allocated by the call.
//
// Order inside a bin: ascending element id, as cil_bins reports it. It comes out of a stable
// LSD radix sort of the bin keys (keys are produced in element order): one pass of 10-bit
// digits when the grid has at most 1024 bins, two passes otherwise. Each pass is a per-tile
// digit histogram (the first with the keys), one exclusive scan over (digit, tile), and a scatter in
// which each tile ranks its elements stably with warp ballots. The work is linear in the element count
// whatever the bin occupancy; a grid collapsed to one bin costs the same as any other. Bound by
// latency (20 MB move for 1M elements): a tile is shared by eight warps, each ranking its part against
// its own counters, and the launches overlap (launch_step). 1M elements in 0.46M bins: 58 us a call;
// with one warp per tile and 14 launches 145 us.
//
// Limits: at most kMaxElems elements and kMaxBins bins per call (about 14.7 MB of scratch,
// held by every GPU that loads the library until the process exits).
//
// Set-up: the first call on a device looks up the arrays' device addresses with
// cudaGetSymbolAddress (with that device current) and caches them; make that first call
// before any stream capture. Every call shares the same scratch, so calls whose work
// overlaps on the GPU race and must be serialised by the caller (one stream, or events).
// Each call clears or overwrites every scratch word it reads before it runs, so the contents
// left by the previous call do not matter.
#include <cuda_runtime.h>

#include <mutex>

#include "cil_internal.cuh"

namespace cil {
namespace {

constexpr int kMaxElems = 1 << 20;
constexpr int kMaxBins = 1 << 20;
constexpr int kNaTile = 256;
constexpr int kNaScan = 1024;        // entries per scan block
constexpr int kDigitBits = 10;       // radix digit: 1024 buckets
constexpr int kDigits = 1 << kDigitBits;
constexpr int kRadixTile = 2048;     // elements per radix tile (8 warps, 8 chunks of 32 each)
constexpr int kRadixWarps = kNaTile / 32;
constexpr int kRadixChunks = kRadixTile / kNaTile;
constexpr int kMaxTiles = kMaxElems / kRadixTile;
constexpr int kIdBits = 20;          // element id field of a packed pass-0 entry (kMaxElems = 2^20)
constexpr int kMaxDevices = 64;
static_assert(kMaxElems <= (1 << kIdBits), "element ids must fit the packed field");
static_assert(kMaxBins <= kDigits * kDigits, "two radix passes must cover every bin key");

static __device__ __align__(256) int g_na_key[kMaxElems];                 // bin key per element
static __device__ __align__(256) int g_na_alt[kMaxElems];                 // pass 0 out: id | high digit << 20
static __device__ __align__(256) int g_na_count[kMaxBins + kNaScan];      // bin counts (+ end sentinel room)
static __device__ __align__(256) int g_na_hist[kDigits * kMaxTiles];      // [digit][tile] counts -> offsets
static __device__ __align__(256) int g_na_part[kMaxBins / kNaScan + 1];   // scan partials (bin counts)
static __device__ __align__(256) int g_na_part_hist[kMaxTiles];           // scan partials (first histogram)

struct Scratch {
  int *key;
  int *alt;
  int *count;
  int *hist;
  int *part;
  int *part_hist;
};

struct NaGeom {
  int dim;
  int ns[3];
  double ih[3];
  float scale[3];  // ns / L
};

__global__ void k_na_clear(int *count, int nbins_pad) {
  enter_step_kernel();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nbins_pad; i += gridDim.x * blockDim.x) count[i] = 0;
}

// per radix tile: the elements' bins, the bin counts, and the histogram of the first pass's digits,
// written digit-major (hist[digit * ntiles + tile]) so that one exclusive scan gives every (digit, tile)
// its first output position
__global__ void __launch_bounds__(kNaTile) k_na_keys(const double *__restrict__ pos, int n, NaGeom g, int ntiles, int *key,
                                                     int *count, int *hist) {
  enter_step_kernel();
  __shared__ int h[kDigits];
  for (int d = threadIdx.x; d < kDigits; d += kNaTile) h[d] = 0;
  __syncthreads();
  const int e0 = blockIdx.x * kRadixTile + threadIdx.x;
#pragma unroll
  for (int q = 0; q < kRadixChunks; ++q) {
    const int e = e0 + q * kNaTile;
    if (e >= n) continue;
    int ls[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (d >= g.dim) continue;
      const double x = pos[static_cast<size_t>(e) * g.dim + d];
      int v = floor_scaled(x, g.scale[d], [&] { return __dmul_rn(__dmul_rn(x, g.ih[d]), static_cast<double>(g.ns[d])); });
      v = v < g.ns[d] - 1 ? v : g.ns[d] - 1;
      ls[d] = v > 0 ? v : 0;
    }
    const int b = g.dim == 2 ? ls[0] * g.ns[1] + ls[1] : (ls[0] * g.ns[1] + ls[1]) * g.ns[2] + ls[2];
    key[e] = b;
    atomicAdd(count + b, 1);
    atomicAdd(h + (b & (kDigits - 1)), 1);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kDigits; d += kNaTile) hist[d * ntiles + blockIdx.x] = h[d];
}

__device__ __forceinline__ int na_block_scan(int v, int *total) {
  __shared__ int ws[kNaTile / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) ws[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    int w = lane < kNaTile / 32 ? ws[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    if (lane < kNaTile / 32) ws[lane] = w;
  }
  __syncthreads();
  const int base = wid > 0 ? ws[wid - 1] : 0;
  *total = ws[kNaTile / 32 - 1];
  __syncthreads();
  return base + inc - v;
}

// sums of the scan blocks (kNaScan entries) of a (na blocks, sums to pa) and of b (the other blocks, to pb)
__global__ void __launch_bounds__(kNaTile) k_na_partial(const int *a, int na, int *pa, const int *b, int *pb) {
  enter_step_kernel();
  const bool first = static_cast<int>(blockIdx.x) < na;
  const int blk = first ? blockIdx.x : blockIdx.x - na;
  const int4 v = reinterpret_cast<const int4 *>((first ? a : b) + blk * kNaScan)[threadIdx.x];
  int tot;
  na_block_scan(v.x + v.y + v.z + v.w, &tot);
  if (threadIdx.x == 0) (first ? pa : pb)[blk] = tot;
}

// the sum of the scan blocks before blk (at most about 1000: a few loads per thread)
__device__ __forceinline__ int na_before(const int *part, int blk) {
  int v = 0, tot;
  for (int i = threadIdx.x; i < blk; i += kNaTile) v += part[i];
  na_block_scan(v, &tot);
  return tot;
}

// blocks below na: bin starts from the bin counts; the others: in-place exclusive scan of the (digit,
// tile) counts
__global__ void __launch_bounds__(kNaTile) k_na_offsets(const int *count, int na, const int *pa, int nbins, int *bin_start,
                                                        int *hist, const int *ph) {
  enter_step_kernel();
  const bool bins = static_cast<int>(blockIdx.x) < na;
  const int blk = bins ? blockIdx.x : blockIdx.x - na;
  const int before = na_before(bins ? pa : ph, blk);
  int4 *p = reinterpret_cast<int4 *>(const_cast<int *>(bins ? count : hist) + blk * kNaScan) + threadIdx.x;
  const int4 v = *p;
  int tot;
  int s = before + na_block_scan(v.x + v.y + v.z + v.w, &tot);
  if (!bins) {
    *p = make_int4(s, s + v.x, s + v.x + v.y, s + v.x + v.y + v.z);
    return;
  }
  const int b0 = blk * kNaScan + threadIdx.x * 4;
  const int c[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int b = b0 + q;
    if (b <= nbins) bin_start[b] = s;  // bins past nbins are empty: bin_start[nbins] = n
    s += c[q];
  }
}

// radix digit of a word in pass `pass` (0: low 10 bits of the key, 1: high 10 bits, read from the
// packed pass-0 output)
__device__ __forceinline__ int na_digit(int pass, int v) { return pass == 0 ? (v & (kDigits - 1)) : (v >> kIdBits); }

// per radix tile: the second pass's digit histogram
__global__ void __launch_bounds__(kNaTile) k_na_hist(const int *src, int n, int ntiles, int *hist) {
  enter_step_kernel();
  __shared__ int h[kDigits];
  for (int d = threadIdx.x; d < kDigits; d += kNaTile) h[d] = 0;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kRadixChunks; ++q) {
    const int i = blockIdx.x * kRadixTile + q * kNaTile + threadIdx.x;
    if (i < n) atomicAdd(h + na_digit(1, src[i]), 1);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kDigits; d += kNaTile) hist[d * ntiles + blockIdx.x] = h[d];
}

// Per radix tile, each warp takes kRadixChunks x 32 consecutive elements: an element's rank among
// those of its digit in the warp's part (ballots + popcount over the warp's own counters, in element
// order), then the warps' counters become their first places (the (digit, tile) offset plus the earlier
// warps' counts), so the scatter is stable. Pass 0 of two writes id | high digit << 20 into alt; the
// last pass writes element ids into the caller's array.
__global__ void __launch_bounds__(kNaTile) k_na_rank_scatter(int pass, int last, const int *src, int n, int ntiles,
                                                             const int *hist, int *alt, int *elems) {
  enter_step_kernel();
  __shared__ int cur[kRadixWarps][kDigits];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i0 = blockIdx.x * kRadixTile + w * (kRadixChunks * 32) + lane;
  int v[kRadixChunks], rank[kRadixChunks];
#pragma unroll
  for (int q = 0; q < kRadixChunks; ++q) v[q] = i0 + q * 32 < n ? src[i0 + q * 32] : -1;
  for (int d = lane; d < kDigits; d += 32) cur[w][d] = 0;
  __syncwarp();
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int q = 0; q < kRadixChunks; ++q) {
    const bool valid = i0 + q * 32 < n;
    const int d = valid ? na_digit(pass, v[q]) : 0;
    // the lanes of the same digit, bit by bit (a warp match takes a round per distinct value, and most
    // digits of a chunk are distinct)
    unsigned peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < kDigitBits; ++b) {
      const unsigned m = __ballot_sync(0xffffffffu, (d >> b) & 1);
      peers &= (d >> b) & 1 ? m : ~m;
    }
    const int at = valid ? cur[w][d] : 0;  // every lane reads before any leader advances
    __syncwarp();
    if (valid && lane == __ffs(peers) - 1) cur[w][d] = at + __popc(peers);
    __syncwarp();
    rank[q] = at + __popc(peers & lt);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kDigits; d += kNaTile) {
    int off = hist[d * ntiles + blockIdx.x];
#pragma unroll
    for (int k = 0; k < kRadixWarps; ++k) {
      const int c = cur[k][d];
      cur[k][d] = off;
      off += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kRadixChunks; ++q) {
    const int i = i0 + q * 32;
    if (i >= n) continue;
    const int at = cur[w][na_digit(pass, v[q])] + rank[q];
    const int id = pass == 0 ? i : (v[q] & ((1 << kIdBits) - 1));
    if (last)
      elems[at] = id;
    else
      alt[at] = id | ((v[q] >> kDigitBits) << kIdBits);
  }
}

std::mutex g_na_mutex;
bool g_na_ready[kMaxDevices] = {};
Scratch g_na_scratch[kMaxDevices];

cil_status na_scratch(int dev, Scratch *out) {
  if (dev < 0 || dev >= kMaxDevices) return CIL_ERR_CONFIG;
  std::lock_guard<std::mutex> lock(g_na_mutex);
  if (!g_na_ready[dev]) {
    Scratch s{};
    if (cudaGetSymbolAddress(reinterpret_cast<void **>(&s.key), g_na_key) != cudaSuccess ||
        cudaGetSymbolAddress(reinterpret_cast<void **>(&s.alt), g_na_alt) != cudaSuccess ||
        cudaGetSymbolAddress(reinterpret_cast<void **>(&s.count), g_na_count) != cudaSuccess ||
        cudaGetSymbolAddress(reinterpret_cast<void **>(&s.hist), g_na_hist) != cudaSuccess ||
        cudaGetSymbolAddress(reinterpret_cast<void **>(&s.part), g_na_part) != cudaSuccess ||
        cudaGetSymbolAddress(reinterpret_cast<void **>(&s.part_hist), g_na_part_hist) != cudaSuccess)
      return CIL_ERR_CUDA;
    g_na_scratch[dev] = s;
    g_na_ready[dev] = true;
  }
  *out = g_na_scratch[dev];
  return CIL_OK;
}

}  // namespace
}  // namespace cil

extern "C" cil_status cil_bin_elements_noalloc(const double *pos, int32_t n_elems, int32_t dim,
                                               const double *box, double width, int32_t *ns,
                                               int32_t *bin_start, int32_t *elems, int32_t max_bins,
                                               void *stream) {
  using namespace cil;
  if (!pos || !box || !ns || !bin_start || !elems || (dim != 2 && dim != 3) || n_elems < 0 ||
      !(width > 0.0))
    return CIL_ERR_CONFIG;
  if (n_elems > kMaxElems) return CIL_ERR_CAPACITY;
  // grid of LinkListOrtho::get_opt_size + reset (Utils.hpp:872-908)
  NaGeom g{};
  g.dim = dim;
  double mn = box[0];
  for (int d = 1; d < dim; ++d) mn = mn < box[d] ? mn : box[d];
  const double ir = 1.0 / (width + mn * 1.0e-8);
  bool collapse = false;
  long long nb = 1;
  for (int d = 0; d < 3; ++d) {
    g.ns[d] = 1;
    g.ih[d] = 0.0;
  }
  for (int d = 0; d < dim; ++d) {
    if (!(box[d] > 0.0)) return CIL_ERR_CONFIG;
    // more than kMaxBins bins along one axis never fit (and would overflow the int cast)
    if (!(box[d] * ir < static_cast<double>(kMaxBins) + 1.0)) return CIL_ERR_CAPACITY;
    g.ns[d] = static_cast<int>(box[d] * ir);
    g.ih[d] = 1.0 / box[d];
    collapse = collapse || g.ns[d] < 3;
  }
  if (collapse)
    for (int d = 0; d < dim; ++d) g.ns[d] = 1;
  for (int d = 0; d < dim; ++d) nb *= g.ns[d];
  for (int d = 0; d < 3; ++d) g.scale[d] = static_cast<float>(g.ih[d] * g.ns[d]);
  for (int d = 0; d < 3; ++d) ns[d] = g.ns[d];
  if (nb > kMaxBins || nb > max_bins) return CIL_ERR_CAPACITY;
  const int nbins = static_cast<int>(nb);
  const int nparts = (nbins + 1 + kNaScan - 1) / kNaScan;  // room for the end sentinel
  const int nbins_pad = nparts * kNaScan;                   // <= kMaxBins + kNaScan

  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return CIL_ERR_CUDA;
  Scratch sc{};
  cil_status st = na_scratch(dev, &sc);
  if (st != CIL_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int ntiles = (n_elems + kRadixTile - 1) / kRadixTile;
  const int hparts = ntiles;  // kDigits * ntiles entries, kNaScan per scan block
  launch_step(false, (nbins_pad + kNaTile - 1) / kNaTile, kNaTile, 0, s, k_na_clear, sc.count, nbins_pad);  // after the caller's work
  if (n_elems > 0) launch_step(true, ntiles, kNaTile, 0, s, k_na_keys, pos, n_elems, g, ntiles, sc.key, sc.count, sc.hist);
  launch_step(true, nparts + hparts, kNaTile, 0, s, k_na_partial, sc.count, nparts, sc.part, sc.hist, sc.part_hist);
  launch_step(true, nparts + hparts, kNaTile, 0, s, k_na_offsets, sc.count, nparts, sc.part, nbins, bin_start, sc.hist,
              sc.part_hist);
  if (n_elems > 0) {
    // stable radix sort of the keys by bin: one pass of 10-bit digits for grids of at most
    // 1024 bins, two otherwise (ntiles <= 512, so the histogram scan has <= 512 blocks)
    const int npass = nbins <= kDigits ? 1 : 2;
    launch_step(true, ntiles, kNaTile, 0, s, k_na_rank_scatter, 0, npass == 1, sc.key, n_elems, ntiles, sc.hist, sc.alt,
                elems);
    if (npass == 2) {
      launch_step(true, ntiles, kNaTile, 0, s, k_na_hist, sc.alt, n_elems, ntiles, sc.hist);
      launch_step(true, hparts, kNaTile, 0, s, k_na_partial, sc.hist, hparts, sc.part, sc.hist, sc.part);
      launch_step(true, hparts, kNaTile, 0, s, k_na_offsets, sc.count, 0, sc.part, nbins, bin_start, sc.hist, sc.part);
      launch_step(true, ntiles, kNaTile, 0, s, k_na_rank_scatter, 1, 1, sc.alt, n_elems, ntiles, sc.hist, sc.alt, elems);
    }
  }
  if (cudaGetLastError() != cudaSuccess) return CIL_ERR_CUDA;
  return CIL_OK;
}
