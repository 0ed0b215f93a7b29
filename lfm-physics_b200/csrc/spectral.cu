// S_a Helmholtz filter fused with the transforms along the slowest axis.
//
// The reference smooths each colour's |Psi_a|^2 as
//   S_a = IRFFT3[ gamma / (gamma + D |k|^2) * RFFT3(|Psi_a|^2) ]
// (lfm/core/backends/numpy_backend.py:341-356).  A 3-D transform is three 1-D
// passes, so the solve is split as
//   2-D R2C over (j, k) for every plane i and colour (cuFFT, or in one CTA: below)
//   -> this kernel: forward 1-D FFT along i, times the filter, inverse 1-D FFT
//   -> 2-D C2R over (j, k).
// This kernel replaces three HBM round trips of the half spectrum (the forward
// pass along i, the filter multiply, the inverse pass along i) by one.
//
// Spectrum layout (cuFFT's R2C output): spec[a][x][w], w = y * (N/2+1) + z,
// so for a fixed x the columns w are contiguous.  A CTA owns TW consecutive
// columns of one colour and all N values of x in each.  The length-N FFT of a
// column is the four-step factorisation N = N1 * N2 (Bailey's "four-step FFT",
// also in Van Loan, Computational Frameworks for the FFT, 3.3): thread n1 of a
// column holds x[n1 + N1 m] (m < N2); a length-N2 DFT in registers, a twiddle
// w_N^(n1 k2), an exchange through shared memory, a length-N1 DFT in
// registers; the inverse retraces the steps with conjugate twiddles, so every
// thread ends with the elements it loaded.  The register DFTs are iterative
// radix-2 Cooley-Tukey (decimation in time).  Twiddles w_N^j = e^{-2 pi i j/N}
// come from tables computed on the host in double precision: the length-N
// table in shared memory for the twiddles between the two DFTs, and the
// length-32 table in constant memory for the register DFTs (M <= 32).
//
// The filter factor of each spectral point, gamma/(gamma + D k^2) / N^3
// rounded to float32 once, is read from a table over (|fx|, |fy|, fz) built by
// helmholtz_table_kernel with the float64 arithmetic of NumPy's filter
// (k = 2 pi fftfreq(N)); k^2 depends only on the magnitudes of the integer
// frequencies, so (N/2+1)^3 entries cover the spectrum.
#include "lfm_kernels.h"
#include "lfm_launch.h"

#include <cmath>

namespace lfm {
namespace {

__host__ __device__ constexpr int bitrev(int i, int bits) {
  int r = 0;
  for (int b = 0; b < bits; ++b) r |= ((i >> b) & 1) << (bits - 1 - b);
  return r;
}
__host__ __device__ constexpr int log2i(int n) { return n <= 1 ? 0 : 1 + log2i(n / 2); }

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)),
                     __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }

// e^{-2 pi i t / 32}, t < 32: the twiddles of the register DFTs (M <= 32),
// w_M^u = c_w32[u * 32 / M].  The indices are compile-time constants, so each
// twiddle is an operand from the constant bank, not a shared-memory load.
// The values equal the pass's own table (e^{-2 pi i (u N / M) / N} has the same
// angle u / M in double).
__constant__ float2 c_w32[32];

// One radix-2 stage (butterflies of span LEN / 2) of an in-register DFT of
// size M; a[] is in bit-reversed order before the first stage.
template <int M, int LEN, bool INV>
__device__ __forceinline__ void dft_stage(float2 (&a)[M]) {
  static_assert(M <= 32, "register DFTs take their twiddles from c_w32");
  constexpr int half = LEN / 2, step = M / LEN;
#pragma unroll
  for (int i = 0; i < M; i += LEN) {
#pragma unroll
    for (int j = 0; j < half; ++j) {
      const int u = j * step;  // exponent in units of w_M
      float2 t = a[i + j + half];
      if (u == 0) {
      } else if (4 * u == M) {  // w_M^(M/4) = -i (forward), +i (inverse)
        t = INV ? make_float2(-t.y, t.x) : make_float2(t.y, -t.x);
      } else {
        const float2 w = c_w32[u * (32 / M)];
        t = cmul(t, INV ? conjf2(w) : w);
      }
      const float2 s = a[i + j];
      a[i + j] = make_float2(s.x + t.x, s.y + t.y);
      a[i + j + half] = make_float2(s.x - t.x, s.y - t.y);
    }
  }
  if constexpr (LEN < M) dft_stage<M, 2 * LEN, INV>(a);
}

// v[k] <- sum_j v[j] w_M^(s j k), s = -1 (forward, e^{-}) or +1 (inverse), in
// registers.
template <int M, bool INV>
__device__ __forceinline__ void dft_reg(float2 (&v)[M]) {
  constexpr int B = log2i(M);
  float2 a[M];
#pragma unroll
  for (int i = 0; i < M; ++i) a[bitrev(i, B)] = v[i];
  dft_stage<M, 2, INV>(a);
#pragma unroll
  for (int i = 0; i < M; ++i) v[i] = a[i];
}

// One CTA: TW columns w0 .. w0+TW-1 of colour a.  Thread (n1, c), n1 < N1,
// c < TW, tid = n1 * TW + c.  Shared exchange buffer S(c, n1, k2) at
// (k2 * N1 + n1) * TW + c: consecutive threads touch consecutive columns in
// every phase (two 8-byte wavefronts per warp, no further conflicts).
template <int N1, int N2, int TW>
__global__ void __launch_bounds__(N1* TW) helmholtz_xpass_kernel(float2* __restrict__ spec,
                                                                 const float* __restrict__ table,
                                                                 const float2* __restrict__ twg) {
  constexpr int N = N1 * N2;
  constexpr int H = N / 2 + 1;
  constexpr int64_t W = (int64_t)N * H;  // columns per colour
  constexpr int G = N2 / N1;             // k2 groups per thread after the exchange
  static_assert(N2 % N1 == 0, "N2 must be a multiple of N1");
  extern __shared__ float2 smem_x[];
  float2* tw = smem_x;      // N twiddles
  float2* S = smem_x + N;   // N * TW exchange buffer
  const int tid = threadIdx.x;
  const int n1 = tid / TW, c = tid % TW;
  for (int t = tid; t < N; t += N1 * TW) tw[t] = twg[t];
  const int64_t tiles_per_colour = W / TW;
  const int a = (int)(blockIdx.x / tiles_per_colour);
  const int64_t w = (blockIdx.x % tiles_per_colour) * TW + c;
  float2* col = spec + (int64_t)a * N * W + w;  // element x at col[x * W]
  const int y = (int)(w / H), z = (int)(w % H);
  const int fy = y <= N - y ? y : N - y;
  const float* trow = table + (int64_t)fy * H + z;  // + |fx| * H * H
  __syncthreads();  // twiddles

  // ---- forward along x -------------------------------------------------------
  float2 v[N2];
#pragma unroll
  for (int m = 0; m < N2; ++m) v[m] = col[(int64_t)(n1 + N1 * m) * W];
  dft_reg<N2, false>(v);  // v[k2] = Y[n1][k2]
#pragma unroll
  for (int k2 = 1; k2 < N2; ++k2) v[k2] = cmul(v[k2], tw[n1 * k2]);
#pragma unroll
  for (int k2 = 0; k2 < N2; ++k2) S[(k2 * N1 + n1) * TW + c] = v[k2];
  __syncthreads();
  float2 u[G][N1];  // group g: k2 = n1 + N1 g (this thread's k2 values)
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const int k2 = n1 + N1 * g;
#pragma unroll
    for (int j = 0; j < N1; ++j) u[g][j] = S[(k2 * N1 + j) * TW + c];
    dft_reg<N1, false>(u[g]);  // u[g][k1] = X[k2 + N2 k1]
    // ---- the filter --------------------------------------------------------
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
      const int k = k2 + N2 * k1;
      const int fx = k <= N - k ? k : N - k;
      const float f = __ldg(trow + (int64_t)fx * H * H);
      u[g][k1] = make_float2(u[g][k1].x * f, u[g][k1].y * f);
    }
    // ---- inverse along x, first half ---------------------------------------
    dft_reg<N1, true>(u[g]);  // u[g][j] = sum_k1 X w_N1^(-k1 j)
#pragma unroll
    for (int j = 1; j < N1; ++j) u[g][j] = cmul(u[g][j], conjf2(tw[k2 * j]));
  }
  __syncthreads();  // every thread has read S
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const int k2 = n1 + N1 * g;
#pragma unroll
    for (int j = 0; j < N1; ++j) S[(k2 * N1 + j) * TW + c] = u[g][j];
  }
  __syncthreads();
#pragma unroll
  for (int k2 = 0; k2 < N2; ++k2) v[k2] = S[(k2 * N1 + n1) * TW + c];
  dft_reg<N2, true>(v);  // v[m] = x[n1 + N1 m] (times N: unnormalised)
#pragma unroll
  for (int m = 0; m < N2; ++m) col[(int64_t)(n1 + N1 * m) * W] = v[m];
}

// ---- 2-D transforms of a plane in one CTA (N = 64, 128) ------------------------
//
// cuFFT takes two kernels for the 2-D transform of these planes, each a pass over the
// data and a launch.  A plane (16 or 64 KB) fits into shared memory, so one CTA does
// both directions of it: rows two at a time as the real and imaginary part of one
// complex transform, columns 0 and N/2 of the half spectrum (real for every row) as one
// column in the same way.  That leaves N/2 complex transforms of length N each way,
// N1 threads with N2 elements each (the four-step scheme above).  Whole COLOR steps with
// S_a: 64^3 32.0 -> 28.2 us, 128^3 157 -> 153 (there the stencil takes 91).  A plane of
// 256^2 (264 KB) does not fit and stays with cuFFT.
template <int N1, int N2>
struct PlaneShape {
  static constexpr int N = N1 * N2, H = N / 2, G = N2 / N1, T = H * N1;
  // a row transform's exchange rows, padded so that neighbouring transforms start on
  // other banks; a half-spectrum row, padded for the row-wise accesses
  static constexpr int LE = N + N1, LS = H + 1;
  static constexpr int kSmem = (N + (H * LE > N * H ? H * LE : N * H) + N * LS + N) * 8;
};

// A length-N transform, N1 threads each: v[m] is element n1 + N1 m; at(q): the
// exchange place of element q of this transform; the thread ends with X[k2 + N2 k1],
// k2 = n1 + N1 g, in u[g][k1].
template <int N1, int N2, bool INV, class At>
__device__ __forceinline__ void fft_split(float2 (&v)[N2], float2 (&u)[N2 / N1][N1], int n1,
                                          const float2* tw, const At& at) {
  dft_reg<N2, INV>(v);
#pragma unroll
  for (int k2 = 1; k2 < N2; ++k2) {
    const float2 w = tw[n1 * k2];
    v[k2] = cmul(v[k2], INV ? conjf2(w) : w);
  }
#pragma unroll
  for (int k2 = 0; k2 < N2; ++k2) *at(k2 * N1 + n1) = v[k2];
  __syncthreads();
#pragma unroll
  for (int g = 0; g < N2 / N1; ++g) {
#pragma unroll
    for (int j = 0; j < N1; ++j) u[g][j] = *at((n1 + N1 * g) * N1 + j);
    dft_reg<N1, INV>(u[g]);
  }
}

// spec[plane][y][z] <- the 2-D real transform of real[plane][j][k].
template <int N1, int N2>
__global__ void __launch_bounds__(N1* N1* N2 / 2) plane_r2c_kernel(const float* __restrict__ real,
                                                                   float2* __restrict__ spec,
                                                                   const float2* __restrict__ twg) {
  using P = PlaneShape<N1, N2>;
  constexpr int N = P::N, H = P::H;
  extern __shared__ float2 smem_p[];
  float2* tw = smem_p;
  float2* S = tw + N;          // N x LS half spectrum after the rows
  float2* C = S + N * P::LS;   // column 0
  float2* E = C + N;           // exchange
  const int tid = threadIdx.x;
  for (int t = tid; t < N; t += P::T) tw[t] = twg[t];
  const float* in = real + (int64_t)blockIdx.x * N * N;
  float2* out = spec + (int64_t)blockIdx.x * N * (H + 1);
  float2 v[N2], u[P::G][N1];
  {  // rows 2 p and 2 p + 1
    const int p = tid / N1, n1 = tid % N1;
    const float *ra = in + 2 * p * N, *rb = ra + N;
#pragma unroll
    for (int m = 0; m < N2; ++m) v[m] = make_float2(ra[n1 + N1 * m], rb[n1 + N1 * m]);
    __syncthreads();  // twiddles
    fft_split<N1, N2, false>(v, u, n1, tw, [&](int q) { return E + p * P::LE + q; });
    __syncthreads();
#pragma unroll
    for (int g = 0; g < P::G; ++g)
#pragma unroll
      for (int k1 = 0; k1 < N1; ++k1) E[p * P::LE + n1 + N1 * g + N2 * k1] = u[g][k1];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < N2 / 2; ++m) {  // Z[k] = A[k] + i B[k] taken apart
      const int k = n1 + N1 * m;
      const float2 z = E[p * P::LE + k], w = E[p * P::LE + (k ? N - k : H)];
      float2 a, b;
      if (k == 0) {  // columns 0 and N/2, both real, as one
        a = make_float2(z.x, w.x);
        b = make_float2(z.y, w.y);
      } else {
        a = make_float2(0.5f * (z.x + w.x), 0.5f * (z.y - w.y));
        b = make_float2(0.5f * (z.y + w.y), 0.5f * (w.x - z.x));
      }
      S[2 * p * P::LS + k] = a;
      S[(2 * p + 1) * P::LS + k] = b;
    }
    __syncthreads();
  }
  const int c = tid % H, n1 = tid / H;  // column c
#pragma unroll
  for (int m = 0; m < N2; ++m) v[m] = S[(n1 + N1 * m) * P::LS + c];
  fft_split<N1, N2, false>(v, u, n1, tw, [&](int q) { return E + q * H + c; });
#pragma unroll
  for (int g = 0; g < P::G; ++g)
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
      const int y = n1 + N1 * g + N2 * k1;
      if (c)
        out[y * (H + 1) + c] = u[g][k1];
      else
        C[y] = u[g][k1];
    }
  __syncthreads();
  for (int y = tid; y < N; y += P::T) {
    const float2 z = C[y], w = C[y ? N - y : 0];
    out[y * (H + 1)] = make_float2(0.5f * (z.x + w.x), 0.5f * (z.y - w.y));
    out[y * (H + 1) + H] = make_float2(0.5f * (z.y + w.y), 0.5f * (w.x - z.x));
  }
}

// real[plane][j][k] <- the (unnormalised) inverse of spec[plane][y][z].
template <int N1, int N2>
__global__ void __launch_bounds__(N1* N1* N2 / 2) plane_c2r_kernel(const float2* __restrict__ spec,
                                                                   float* __restrict__ real,
                                                                   const float2* __restrict__ twg) {
  using P = PlaneShape<N1, N2>;
  constexpr int N = P::N, H = P::H;
  extern __shared__ float2 smem_p[];
  float2* tw = smem_p;
  float2* S = tw + N;
  float2* E = S + N * P::LS + N;
  const int tid = threadIdx.x;
  for (int t = tid; t < N; t += P::T) tw[t] = twg[t];
  const float2* in = spec + (int64_t)blockIdx.x * N * (H + 1);
  float* out = real + (int64_t)blockIdx.x * N * N;
  float2 v[N2], u[P::G][N1];
  {
    const int c = tid % H, n1 = tid / H;
#pragma unroll
    for (int m = 0; m < N2; ++m) {
      const float2* row = in + (n1 + N1 * m) * (H + 1);
      v[m] = row[c];
      if (c == 0) {  // F0 + i F(N/2): both columns' inverses are real
        const float2 h = row[H];
        v[m] = make_float2(v[m].x - h.y, v[m].y + h.x);
      }
    }
    __syncthreads();  // twiddles
    fft_split<N1, N2, true>(v, u, n1, tw, [&](int q) { return E + q * H + c; });
#pragma unroll
    for (int g = 0; g < P::G; ++g)
#pragma unroll
      for (int k1 = 0; k1 < N1; ++k1) S[(n1 + N1 * g + N2 * k1) * P::LS + c] = u[g][k1];
    __syncthreads();
  }
  const int p = tid / N1, n1 = tid % N1;
#pragma unroll
  for (int m = 0; m < N2; ++m) {  // Z[k] = A[k] + i B[k] from the half spectra
    const int k = n1 + N1 * m, q = k < H ? k : (k == H ? 0 : N - k);
    const float2 a = S[2 * p * P::LS + q], b = S[(2 * p + 1) * P::LS + q];
    if (k == 0)
      v[m] = make_float2(a.x, b.x);
    else if (k == H)
      v[m] = make_float2(a.y, b.y);
    else if (k < H)
      v[m] = make_float2(a.x - b.y, a.y + b.x);
    else
      v[m] = make_float2(a.x + b.y, b.x - a.y);
  }
  fft_split<N1, N2, true>(v, u, n1, tw, [&](int q) { return E + p * P::LE + q; });
#pragma unroll
  for (int g = 0; g < P::G; ++g)
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
      const int k = n1 + N1 * g + N2 * k1;
      out[2 * p * N + k] = u[g][k1].x;
      out[(2 * p + 1) * N + k] = u[g][k1].y;
    }
}

template <int N1, int N2>
cudaError_t launch_planes(bool inverse, float* real, float2* spec, const float2* tw,
                          cudaStream_t stream) {
  using P = PlaneShape<N1, N2>;
  const void* kernel = inverse ? (const void*)plane_c2r_kernel<N1, N2>
                               : (const void*)plane_r2c_kernel<N1, N2>;
  if (P::kSmem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         P::kSmem);
    if (e != cudaSuccess) return e;
  }
  if (inverse)
    plane_c2r_kernel<N1, N2><<<3 * P::N, P::T, P::kSmem, stream>>>(spec, real, tw);
  else
    plane_r2c_kernel<N1, N2><<<3 * P::N, P::T, P::kSmem, stream>>>(real, spec, tw);
  return cudaGetLastError();
}

// np.fft.fftfreq(n) * 2*pi for the frequency magnitude f: f * (1.0/n) * 2*pi in
// float64 (the sign of f does not change k^2).
__device__ __forceinline__ double wave(int f, int n) {
  return __dmul_rn(__dmul_rn((double)f, 1.0 / (double)n), 2.0 * 3.141592653589793);
}

// table[(fx * H + fy) * H + fz] = float32(gamma / (gamma + D k^2) / N^3), the
// same float64 operations (and the same rounding) as a per-element filter.
__global__ void helmholtz_table_kernel(float* __restrict__ table, int N, double gamma,
                                       double d) {
  const int H = N / 2 + 1;
  const int64_t total = (int64_t)H * H * H;
  const double inv_n3 = 1.0 / ((double)N * N * N);
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int fz = (int)(t % H), fy = (int)((t / H) % H), fx = (int)(t / ((int64_t)H * H));
    const double kx = wave(fx, N), ky = wave(fy, N), kz = wave(fz, N);
    const double k_sq = __dadd_rn(__dadd_rn(__dmul_rn(kx, kx), __dmul_rn(ky, ky)),
                                  __dmul_rn(kz, kz));
    const double h = __ddiv_rn(gamma, __dadd_rn(gamma, __dmul_rn(d, k_sq)));
    table[t] = __double2float_rn(__dmul_rn(h, inv_n3));
  }
}

template <int N1, int N2, int TW>
cudaError_t launch_xpass(float2* spec, const float* table, const float2* tw,
                         cudaStream_t stream) {
  constexpr int N = N1 * N2;
  constexpr int smem = (N + N * TW) * (int)sizeof(float2);
  static SmemGrant grant;
  const cudaError_t e = grant.raise((const void*)helmholtz_xpass_kernel<N1, N2, TW>, smem);
  if (e != cudaSuccess) return e;
  const int64_t W = (int64_t)N * (N / 2 + 1);
  const int64_t tiles = 3 * (W / TW);
  helmholtz_xpass_kernel<N1, N2, TW><<<(unsigned)tiles, N1 * TW, smem, stream>>>(spec, table,
                                                                                  tw);
  return cudaGetLastError();
}

}  // namespace

cudaError_t upload_dft_twiddles() {
  float2 w[32];
  for (int t = 0; t < 32; ++t) {
    const double ang = -2.0 * 3.14159265358979323846 * (double)t / 32.0;
    w[t] = make_float2((float)std::cos(ang), (float)std::sin(ang));
  }
  return cudaMemcpyToSymbol(c_w32, w, sizeof(w));
}

bool helmholtz_xpass_supported(int N) {
  return N == 64 || N == 128 || N == 256 || N == 512 || N == 1024;
}

bool plane_transform_supported(int N) { return N == 64 || N == 128; }

cudaError_t launch_plane_transform(bool inverse, float* real, float2* spec, const float2* tw, int N,
                                   cudaStream_t stream) {
  if (N == 64) return launch_planes<8, 8>(inverse, real, spec, tw, stream);
  if (N == 128) return launch_planes<8, 16>(inverse, real, spec, tw, stream);
  return cudaErrorNotSupported;
}

cudaError_t launch_helmholtz_table(float* table, int N, double gamma, double d,
                                   cudaStream_t stream) {
  const int64_t total = (int64_t)(N / 2 + 1) * (N / 2 + 1) * (N / 2 + 1);
  int64_t blocks = (total + 255) / 256;
  if (blocks > 148 * 32) blocks = 148 * 32;
  helmholtz_table_kernel<<<(unsigned)blocks, 256, 0, stream>>>(table, N, gamma, d);
  return cudaGetLastError();
}

cudaError_t launch_helmholtz_xpass(float2* spec, const float* table, const float2* tw, int N,
                                   cudaStream_t stream) {
  switch (N) {
    case 64: return launch_xpass<8, 8, 32>(spec, table, tw, stream);
    case 128: return launch_xpass<8, 16, 32>(spec, table, tw, stream);
    case 256: return launch_xpass<16, 16, 16>(spec, table, tw, stream);
    case 512: return launch_xpass<16, 32, 16>(spec, table, tw, stream);
    case 1024: return launch_xpass<32, 32, 8>(spec, table, tw, stream);
    default: return cudaErrorNotSupported;
  }
}

}  // namespace lfm
