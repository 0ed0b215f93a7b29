// On-device float64 metrics of a lattice state.
//
// Reproduces compute_metrics (lfm/analysis/metrics.py:29-111) apart from
// the cluster count:
//   energy_components (lfm/analysis/energy.py:26-113): per cell, in float64,
//     T = 1/2 sum_comp ((psi - psi_prev)/dt)^2
//     G = 1/2 c^2 sum_comp sum_axis g^2, g = np.gradient (central in the
//         interior, one-sided first differences at the two edges; NOT periodic)
//     V = 1/2 chi^2 sum_comp psi^2
//   chi_statistics / well_fraction / void_fraction over interior_mask
//   (lfm/analysis/structure.py:26-171): dist = sqrt((i-c)^2+(j-c)^2+(k-c)^2)
//   <= c*(1-boundary_fraction) with c = N/2, in float64.
//
// A thread keeps a (j, k) column four cells wide of a chunk of planes and marches
// along i: a plane's values serve as next, centre and previous plane, and come, like
// the j neighbours and the previous field, in 16-byte loads.  The edge weights and
// the factors 1/dt^2, 1/2 c^2 are applied to the sums, and the interior test compares
// the integer key 4 dist^2, so the march has no division, no square root and little
// index arithmetic.  COMPLEX 256^3: 112 us, 3.0 TB/s of the 335 MB read; a pass over
// single cells with all of these per cell took 1060 us, with the march but one cell a
// thread 147.  It waits for loads: neither the conversions to float64 (50 % of their
// pipe) nor float64 arithmetic (23 %) fill up.  The partial rows' sum, with a thread a
// quantity, took 51 us; with a warp each and eight loads in flight, 5.
//
// Each CTA reduces its cells to one row of partials in the scratch buffer; a
// second single-CTA kernel reduces the rows in a fixed order (a warp per quantity),
// so results are deterministic for a given grid.
#include <cmath>
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "lfm_b200.h"
#include "lfm_kernels.h"
#include "lfm_metrics.h"

namespace lfm {
namespace {

struct Acc {
  double s[kMetricSums];
  float mn, mx;
};

constexpr int kThreads = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

// Planes of a march: long enough to amortise its first two planes, short enough
// that a small lattice has work for every SM (COLOR 64^3: 16.6 us with 2 planes,
// 46.7 with 8; COMPLEX 256^3: 123.1 with 2, 112.1 with 8, 117.9 with 16).
int march_planes(int N) { return N <= 64 ? 2 : (N <= 128 ? 4 : 8); }

// V floats at p (16-byte aligned when V is 4: N % 4 == 0 and aligned fields).
template <int V>
__device__ __forceinline__ void load_cells(const float* p, float (&x)[V]) {
  if constexpr (V == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
  } else {
    x[0] = *p;
  }
}

// A thread's column is V cells wide along k.  qmax: largest 4 dist^2 of an interior
// cell (dist <= radius in float64).  PREV: all previous fields are given; a field without
// one adds no kinetic energy, also where it is not finite (v - v is NaN there).  The test
// in the march costs COMPLEX 256^3 25 us, so it is left out where it is not needed.
template <int LEVEL, int V, bool PREV>
__global__ void __launch_bounds__(kThreads, V == 4 ? 2 : (LEVEL == LFM_COLOR ? 2 : 4))
    metrics_partial_kernel(MetricsArgs a, int64_t qmax, int planes, int64_t items,
                           double* partials) {
  constexpr int NC = LEVEL == LFM_REAL ? 1 : (LEVEL == LFM_COMPLEX ? 2 : 6);
  const int N = a.N, n2 = N * N;
  const int64_t n3 = (int64_t)n2 * N;
  const int tiles = (n2 / V + kThreads - 1) / kThreads;
  Acc A;
#pragma unroll
  for (int q = 0; q < kMetricSums; ++q) A.s[q] = 0.0;
  A.mn = __int_as_float(0x7f800000);   // +inf
  A.mx = __int_as_float(0xff800000);   // -inf
  const auto field = [&](const float* re, const float* im, int q) -> const float* {
    const bool second = NC > 1 && q >= NC / 2;
    const float* p = second ? im : re;
    return p ? p + (int64_t)(second ? q - NC / 2 : q) * n3 : nullptr;
  };
  int count = 0, well = 0, above = 0, bad = 0;
  double gi = 0.0, gi_edge = 0.0, g = 0.0;
  for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
    const int tile = (int)(item % tiles);
    const int i0 = (int)(item / tiles) * planes, i1 = min(i0 + planes, N);
    const int y = (tile * kThreads + threadIdx.x) * V;
    if (y >= n2) continue;
    const int j = y / N, k = y - j * N;  // V divides N
    const int jm = j > 0 ? -N : 0, jp = j < N - 1 ? N : 0;
    const bool k_lo = k == 0, k_hi = k + V == N;
    const int64_t qj = (int64_t)(2 * j - N) * (2 * j - N);
    float m[NC][V], c[NC][V];
    double gj = 0.0;
    int64_t x = (int64_t)i0 * n2 + y;
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const float* p = field(a.pr, a.pi, q) + x;
      load_cells<V>(p, c[q]);
      load_cells<V>(i0 > 0 ? p - n2 : p, m[q]);
    }
    for (int i = i0; i < i1; ++i, x += n2) {
      const bool edge = i == 0 || i == N - 1;
      double here[V] = {}, di2 = 0.0;
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        const float* p = field(a.pr, a.pi, q) + x;
        const float* old = field(a.pr_prev, a.pi_prev, q);
        float n[V], o[V], lo[V], hi[V];
        load_cells<V>(p + (i == N - 1 ? 0 : n2), n);
        load_cells<V>(old ? old + x : p, o);
        load_cells<V>(p + jm, lo);
        load_cells<V>(p + jp, hi);
        const float left = p[k_lo ? 0 : -1], right = p[k_hi ? V - 1 : V];
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const double v = (double)c[q][e];
          const double d = v - (double)o[e];
          if (PREV || old) A.s[kKinetic] = fma(d, d, A.s[kKinetic]);
          const double di = (double)n[e] - (double)m[q][e];
          di2 = fma(di, di, di2);
          const double dj = (double)hi[e] - (double)lo[e];
          gj = fma(dj, dj, gj);
          const double dk = (double)(e < V - 1 ? c[q][e + 1] : right) -
                            (double)(e > 0 ? c[q][e - 1] : left);
          // np.gradient: half the central difference inside, one-sided at the edges
          const double wk = (e == 0 && k_lo) || (e == V - 1 && k_hi) ? 1.0 : 0.25;
          g = fma(dk * wk, dk, g);
          here[e] = fma(v, v, here[e]);
        }
#pragma unroll
        for (int e = 0; e < V; ++e) {
          m[q][e] = c[q][e];
          c[q][e] = n[e];
        }
      }
      if (edge)
        gi_edge += di2;
      else
        gi += di2;
      float cf[V];
      load_cells<V>(a.chi + x, cf);
      const int64_t qij = (int64_t)(2 * i - N) * (2 * i - N) + qj;
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const double chi = (double)cf[e];
        A.s[kPsiSq] += here[e];
        A.s[kPotential] = fma(chi * chi, here[e], A.s[kPotential]);
        bad += isfinite(cf[e]) && isfinite(here[e]) ? 0 : 1;
        // interior_mask: dist <= c*(1-bf) with c = N/2 (no half-cell shift)
        const int dk = 2 * (k + e) - N;
        if (qij + (int64_t)dk * dk <= qmax) {
          const double d = chi - a.chi_shift;
          ++count;
          A.s[kChiSum] += d;
          A.s[kChiSq] = fma(d, d, A.s[kChiSq]);
          well += cf[e] < a.well ? 1 : 0;
          above += cf[e] > a.void_thr ? 1 : 0;
          A.mn = fminf(A.mn, cf[e]);
          A.mx = fmaxf(A.mx, cf[e]);
        }
      }
    }
    g = fma(jm != 0 && jp != 0 ? 0.25 : 1.0, gj, g);
  }
  A.s[kGradient] = (0.25 * gi + gi_edge) + g;
  A.s[kKinetic] *= 0.5 / (a.dt * a.dt);
  A.s[kGradient] *= 0.5 * a.c2;
  A.s[kPotential] *= 0.5;
  A.s[kCount] = (double)count;
  A.s[kWell] = (double)well;
  A.s[kVoid] = (double)above;
  A.s[kNonFinite] = (double)bad;
  // block reduction: warps -> shared -> row of partials
  __shared__ double sh[kMetricSums][8];
  __shared__ float shmn[8], shmx[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int q = 0; q < kMetricSums; ++q) {
    const double v = warp_sum(A.s[q]);
    if (lane == 0) sh[q][w] = v;
  }
  const float mn = warp_min(A.mn), mx = warp_max(A.mx);
  if (lane == 0) {
    shmn[w] = mn;
    shmx[w] = mx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double* row = partials + (size_t)blockIdx.x * kPartialStride;
    for (int q = 0; q < kMetricSums; ++q) {
      double t = 0.0;
      for (int ww = 0; ww < nw; ++ww) t += sh[q][ww];
      row[q] = t;
    }
    float bmn = shmn[0], bmx = shmx[0];
    for (int ww = 1; ww < nw; ++ww) {
      bmn = fminf(bmn, shmn[ww]);
      bmx = fmaxf(bmx, shmx[ww]);
    }
    row[kMetricSums] = (double)bmn;
    row[kMetricSums + 1] = (double)bmx;
  }
}

// Sums the rows of partials, a warp per quantity: lane l the rows l, l + 32, ... in
// order, then the lanes in a fixed tree.
__global__ void metrics_finish_kernel(const double* partials, int rows, double* out) {
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool sum = q < kMetricSums, low = q == kMetricSums;
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  double t = sum ? 0.0 : (low ? inf : -inf);
  const auto join = [&](double u, double v) { return sum ? u + v : (low ? fmin(u, v) : fmax(u, v)); };
  for (int r = lane; r < rows; r += 8 * 32) {  // eight rows' loads in flight
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      v[u] = r + 32 * u < rows ? partials[(size_t)(r + 32 * u) * kPartialStride + q] : t;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (r + 32 * u < rows) t = join(t, v[u]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double v = __shfl_down_sync(0xffffffffu, t, o);
    t = join(t, v);
  }
  if (lane == 0) out[q] = t;
}

}  // namespace

cudaError_t launch_metrics(const MetricsArgs& a, double* partials, int rows, double* out,
                           cudaStream_t stream) {
  // the largest integer key q = 4 dist^2 whose float64 distance is inside
  int64_t qmax = (int64_t)(4.0 * a.radius * a.radius);
  while (qmax >= 0 && std::sqrt((double)qmax * 0.25) > a.radius) --qmax;
  while (std::sqrt((double)(qmax + 1) * 0.25) <= a.radius) ++qmax;
  const int planes = march_planes(a.N);
  const int64_t n2 = (int64_t)a.N * a.N, chunks = (a.N + planes - 1) / planes;
  // four cells a thread where every row starts on 16 bytes
  const void* all[] = {a.pr, a.pr_prev, a.pi, a.pi_prev, a.chi};
  bool wide = a.N % 4 == 0;
  for (const void* p : all) wide = wide && (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
  const auto run = [&](auto kernel, int V) {
    kernel<<<rows, kThreads, 0, stream>>>(a, qmax, planes, (n2 / V + kThreads - 1) / kThreads * chunks,
                                          partials);
  };
  const bool prev = a.pr_prev && (a.level == LFM_REAL || a.pi_prev);
  const auto run_level = [&](auto level) {
    constexpr int L = decltype(level)::value;
    if (wide)
      prev ? run(metrics_partial_kernel<L, 4, true>, 4) : run(metrics_partial_kernel<L, 4, false>, 4);
    else
      prev ? run(metrics_partial_kernel<L, 1, true>, 1) : run(metrics_partial_kernel<L, 1, false>, 1);
  };
  if (a.level == LFM_REAL)
    run_level(std::integral_constant<int, LFM_REAL>{});
  else if (a.level == LFM_COMPLEX)
    run_level(std::integral_constant<int, LFM_COMPLEX>{});
  else
    run_level(std::integral_constant<int, LFM_COLOR>{});
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  metrics_finish_kernel<<<1, 32 * kPartialStride, 0, stream>>>(partials, rows, out);
  return cudaGetLastError();
}

}  // namespace lfm

// ---------------------------------------------------------------------------
// Metrics without allocation (lfm_metrics_f64_noalloc).
//
// For callers that cannot allocate device memory: a process whose device
// memory is all held by another allocator (PyTorch's caching allocator can
// leave cudaMalloc failing while it keeps free blocks for itself), or a host
// program that allocates only at start-up and must not call cudaMalloc
// afterwards.  Such callers also hold no lfm_context, which is where
// lfm_metrics_f64 keeps its scratch.
//
// The per-CTA partials live in this file-scope device array instead.  Every
// GPU that loads the library holds it until the process ends:
// (kNoAllocRows + 1) rows x kPartialStride (12) doubles = 196,704 bytes
// (192 KiB).  One CTA reduces each 65536 cells, so a lattice may have at most
// kNoAllocRows * 65536 cells (N <= 512).  Host code must not pass the
// array's name to a kernel: on the host it only stands in for the symbol, and
// the device address comes from cudaGetSymbolAddress, taken once per device
// on the first call made with that device current.  That address belongs to
// the device's primary context (the one the CUDA runtime uses), so calls must
// be made with the primary context current.
// ---------------------------------------------------------------------------
namespace {

constexpr int kNoAllocRows = 2048;
constexpr long long kNoAllocCellsPerRow = 65536;

static __device__ __align__(256) double g_noalloc_partials[(kNoAllocRows + 1) *
                                                           lfm::kPartialStride];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
double* g_noalloc_ptr[kNoAllocMaxDevices] = {nullptr};

int noalloc_scratch(double** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return lfm::abi_cuda_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= kNoAllocMaxDevices)
    return lfm::abi_fail(LFM_ERR_UNSUPPORTED, "device index outside the scratch table");
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    double* p = nullptr;
    e = cudaGetSymbolAddress((void**)&p, g_noalloc_partials);
    if (e != cudaSuccess) return lfm::abi_cuda_fail(e, "cudaGetSymbolAddress(metric scratch)");
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return LFM_OK;
}

}  // namespace

extern "C" int lfm_metrics_f64_noalloc(int level, const float* psi_r, const float* psi_r_prev,
                                       const float* psi_i, const float* psi_i_prev,
                                       const float* chi, int N, double dt, double c,
                                       double boundary_fraction, double well_threshold,
                                       double void_threshold, double* out_host, void* stream) {
  lfm::MetricsArgs a{};
  int rc = lfm::metrics_prepare(level, psi_r, psi_r_prev, psi_i, psi_i_prev, chi, N, dt, c,
                                boundary_fraction, well_threshold, void_threshold, out_host, &a);
  if (rc) return rc;
  const long long cells = (long long)N * N * N;
  const long long rows = (cells + kNoAllocCellsPerRow - 1) / kNoAllocCellsPerRow;
  if (rows > kNoAllocRows) {
    char msg[160];
    snprintf(msg, sizeof msg,
             "N=%d needs %lld partial rows; the static scratch holds %d (lattices up to 512^3)",
             N, rows, kNoAllocRows);
    return lfm::abi_fail(LFM_ERR_CAPACITY, msg);
  }
  double* scratch = nullptr;
  rc = noalloc_scratch(&scratch);
  if (rc) return rc;
  // Every partial row and the final row are written before they are read,
  // so nothing left in the array by an earlier call needs clearing.
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  double* final_row = scratch + (size_t)kNoAllocRows * lfm::kPartialStride;
  cudaError_t e = lfm::launch_metrics(a, scratch, (int)rows, final_row, st);
  if (e != cudaSuccess) return lfm::abi_cuda_fail(e, "metrics launch");
  double r[lfm::kPartialStride];
  e = cudaMemcpyAsync(r, final_row, sizeof r, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return lfm::abi_cuda_fail(e, "metrics readback");
  lfm::metrics_finish(r, a.chi_shift, out_host);
  return LFM_OK;
}
