// Adjoint (reverse-mode) leapfrog step for the REAL and COMPLEX levels.
//
// The forward step (lfm/core/backends/numpy_backend.py:80-205), per cell with
// absorb a = 1 - mask, K = kappa/chi0, L the periodic 19-point Laplacian and
// D_ax f = f[x+e_ax] - f[x-e_ax]:
//
//   P'   = a (2P - P_prev + dt2 (L P - X^2 P))        for P = Pr, Pi
//   P_prev' = a P
//   j    = 1/2 sum_ax (Pr D_ax Pi - Pi D_ax Pr)
//   Q    = Pr^2 + Pi^2 + eps_w j - e0^2               (REAL: E^2 - e0^2)
//   acc  = L X - K X Q - [lambda > 0] 4 lambda X (X^2 - chi0^2)
//   Xn   = 2X - X_prev + dt2 acc,  X' = mask chi0 + a max(Xn, -chi0)
//   X_prev' = X
//
// Given the adjoints of (P', P_prev', X', X_prev') this kernel returns the
// adjoints of (P, P_prev, X, X_prev).  L is symmetric and D_ax is
// antisymmetric, so the transposed stencils are L and -D_ax.  With
// u = a gP', gXn = a gX' [Xn not clamped], gQ = -dt2 gXn K X and
// w = eps_w gQ / 2:
//
//   gP_prev = -u                  gX_prev = -gXn
//   gPr = a gPr_prev' + 2u_r + dt2 L u_r - dt2 X^2 u_r + 2 Pr gQ + w sum D Pi + sum D (w Pi)
//   gPi = a gPi_prev' + 2u_i + dt2 L u_i - dt2 X^2 u_i + 2 Pi gQ - w sum D Pr - sum D (w Pr)
//   gX  = gX_prev' + 2 gXn + dt2 L gXn - dt2 gXn (H'(X) + K Q) - 2 dt2 X (Pr u_r + Pi u_i)
//
// with H'(X) = 4 lambda (3 X^2 - chi0^2).  The clamp test needs Xn, which
// depends on the cell's whole stencil; it is read back from the step's output
// instead: a cell was clamped exactly when X' equals mask chi0 + a (-chi0) in
// the forward's float32 arithmetic (a == 0 cells carry no gradient anyway).
//
// Arithmetic is plain float32 (contractions allowed): the adjoint is not tied
// to the reference bit for bit; its accuracy is checked against float64
// autograd and central differences.
#include "lfm_b200.h"
#include "lfm_index.cuh"
#include "lfm_kernels.h"
#include "lfm_queue.cuh"

namespace lfm {
namespace {

struct AdjArgs {
  int level, N;
  const float *pr, *pi, *chi, *chi_next;
  MaskLut lut;
  const float *g_pr, *g_prp, *g_pi, *g_pip, *g_chi, *g_chip;
  float *o_pr, *o_prp, *o_pi, *o_pip, *o_chi, *o_chip;
  float dt2, K, eps_w, e0_sq, four_lambda, chi0, chi0_sq, neg_chi0;
  int use_lambda;
};

// ---- tiled kernel ----------------------------------------------------------
// A CTA owns a TI x TJ x TK block of cells.  Phase 1 evaluates, once per
// point of the block and its one-cell halo, everything the transposed
// stencils need from a neighbour (a*gP', a*gX'*[not clamped], and at the
// COMPLEX level Pr, Pi, w*Pr, w*Pi), into shared memory.  Phase 2 applies
// the stencils from shared memory: a thread takes two cells of a row (8-byte
// loads, sums in packed pairs) in kPlanes planes, so that a field's plane is read
// once for the planes it borders.  The kernel is bound by issue, about 500
// instructions a COMPLEX cell with one cell a thread and every neighbour loaded
// where it is used (28.4 us at 96^3); now 24.4 us.
constexpr int TI = 4, TJ = 8, TK = 32;
constexpr int kPlanes = TI / 2;  // two halves of the CTA share the block's planes
constexpr int HI = TI + 2, HJ = TJ + 2;
// a shared-memory row: cell -1 at [1], the block's cells at [2] .. [TK + 1], the
// cell after at [TK + 2]
constexpr int HK = TK + 4;
constexpr int HALO = HI * HJ * HK;
constexpr int kThreads = 2 * TJ * TK / 2;

template <int LEVEL>
struct TileSmem {
  static constexpr int NF = (LEVEL == LFM_COMPLEX) ? 7 : 2;
  float f[NF][HALO];  // ur, gx [, ui, pr, pi, wpr, wpi]
};

// What the forward writes to a clamped cell's chi: mask*chi0 + a*(-chi0).
__device__ __forceinline__ float clamp_value(const AdjArgs& A, float m, float a) {
  return fadd(fmul(m, A.chi0), fmul(a, A.neg_chi0));
}

// The transposed (= the) Laplacian of a shared-memory field at two cells of kPlanes
// planes, and the cells themselves.  at: the first cell of the plane before.
__device__ __forceinline__ void lap_pairs(const float* f, int at, F2 (&lap)[kPlanes],
                                          F2 (&ctr)[kPlanes]) {
  QPlane<2> q[kPlanes + 2];
#pragma unroll
  for (int p = 0; p < kPlanes + 2; ++p) {
    const int c = at + p * HJ * HK;
    q[p].m = lds<2>(f, c - HK);
    q[p].z = lds<2>(f, c);
    q[p].p = lds<2>(f, c + HK);
    q[p].zl = f[c - 1];
    q[p].zr = f[c + 2];
    if (p > 0 && p <= kPlanes) {
      q[p].ml = f[c - HK - 1];
      q[p].mr = f[c - HK + 2];
      q[p].pl = f[c + HK - 1];
      q[p].pr = f[c + HK + 2];
    }
  }
  const float third = 1.0f / 3.0f, sixth = 1.0f / 6.0f;
#pragma unroll
  for (int p = 0; p < kPlanes; ++p) {
    const S19 a = q_s19<2>(q[p], q[p + 1], q[p + 2], 0), b = q_s19<2>(q[p], q[p + 1], q[p + 2], 1);
    F2 faces, edges;
    sums19_pair(a, b, faces, edges);
    ctr[p] = pk(a.c, b.c);
    lap[p] = pk(fmaf(third, faces.v.x, fmaf(sixth, edges.v.x, -4.0f * a.c)),
                fmaf(third, faces.v.y, fmaf(sixth, edges.v.y, -4.0f * b.c)));
  }
}

// Sum over the axes of f[x + e] - f[x - e] at the same cells, and the cells.
__device__ __forceinline__ void dsum_pairs(const float* f, int at, F2 (&d)[kPlanes],
                                           F2 (&ctr)[kPlanes]) {
  Vec<2> z[kPlanes + 2];
#pragma unroll
  for (int p = 0; p < kPlanes + 2; ++p) z[p] = lds<2>(f, at + p * HJ * HK);
#pragma unroll
  for (int p = 0; p < kPlanes; ++p) {
    const int c = at + (p + 1) * HJ * HK;
    const Vec<2> m = lds<2>(f, c - HK), n = lds<2>(f, c + HK);
    const float l = f[c - 1], r = f[c + 2];
    const Vec<2>&lo = z[p], &here = z[p + 1], &hi = z[p + 2];
    ctr[p] = pk(here.v[0], here.v[1]);
    const F2 di = fsub(pk(hi.v[0], hi.v[1]), pk(lo.v[0], lo.v[1]));
    const F2 dj = fsub(pk(n.v[0], n.v[1]), pk(m.v[0], m.v[1]));
    const F2 dk = pk(here.v[1] - l, r - here.v[0]);
    d[p] = fadd(fadd(di, dj), dk);
  }
}

// PAIR: a thread's two cells are loaded and stored as one (N even, 8-byte aligned).
// U_IN / U_OUT: g_pr, g_pi, g_chi come in / go out as u_r, u_i and gXn, the products
// the step before (in the chain) needs of them.  A cell works its own out once, where
// the raw form looks the sponge and chi's clamp up for every point of every halo.
template <int LEVEL, bool PAIR, bool U_IN, bool U_OUT>
__global__ void __launch_bounds__(kThreads, 3) adjoint_tile_kernel(const AdjArgs A) {
  extern __shared__ __align__(16) float sm_raw[];
  TileSmem<LEVEL>& S = *reinterpret_cast<TileSmem<LEVEL>*>(sm_raw);
  const int N = A.N;
  const int tiles_k = (N + TK - 1) / TK, tiles_j = (N + TJ - 1) / TJ;
  int t = blockIdx.x;
  const int k0 = (t % tiles_k) * TK;
  t /= tiles_k;
  const int j0 = (t % tiles_j) * TJ;
  const int i0 = (t / tiles_j) * TI;
  const float c_w = -0.5f * A.eps_w * A.K * A.dt2;  // w(y) = c_w X(y) gXn(y)

  // phase 1: point terms of the block and its halo.  A warp takes a row of 32 cells at
  // a time (its i and j once for the warp), then the threads take the two cells beyond
  // each row.
  const auto wrap = [&](int x) { return x < 0 ? x + N : (x >= N ? x - N : x); };
  const auto point = [&](int h, int qij, int64_t row, int gk) {
    const int64_t y = row + gk;
    float ur = __ldg(A.g_pr + y), gx = __ldg(A.g_chi + y), ui = 0.0f;
    if constexpr (LEVEL == LFM_COMPLEX) ui = __ldg(A.g_pi + y);
    if constexpr (!U_IN) {
      const float m = mask_from_q_flat(A.lut, qij + qterm(gk, N));
      const float a = fsub(1.0f, m);
      gx = __ldg(A.chi_next + y) != clamp_value(A, m, a) ? a * gx : 0.0f;
      ur = a * ur;
      ui = a * ui;
    }
    S.f[0][h] = ur;
    S.f[1][h] = gx;
    if constexpr (LEVEL == LFM_COMPLEX) {
      const float pr = __ldg(A.pr + y), pi = __ldg(A.pi + y);
      const float w = c_w * __ldg(A.chi + y) * gx;
      S.f[2][h] = ui;
      S.f[3][h] = pr;
      S.f[4][h] = pi;
      S.f[5][h] = w * pr;
      S.f[6][h] = w * pi;
    }
  };
  // rows and columns past the lattice's end stand for the cells they wrap to: only the
  // first of them is read, so one fold is enough (any further ones stay in range)
  const int lane = threadIdx.x & 31;
  const int gl = min(wrap(k0 + lane), N - 1);
#pragma unroll 2
  for (int r = threadIdx.x >> 5; r < HI * HJ; r += kThreads / 32) {
    const int gi = min(wrap(i0 + r / HJ - 1), N - 1), gj = min(wrap(j0 + r % HJ - 1), N - 1);
    point(r * HK + 2 + lane, qterm(gi, N) + qterm(gj, N), ((int64_t)gi * N + gj) * N, gl);
  }
  if (threadIdx.x < 2 * HI * HJ) {
    const int r = threadIdx.x >> 1, side = threadIdx.x & 1;
    const int gi = min(wrap(i0 + r / HJ - 1), N - 1), gj = min(wrap(j0 + r % HJ - 1), N - 1);
    point(r * HK + (side ? TK + 2 : 1), qterm(gi, N) + qterm(gj, N), ((int64_t)gi * N + gj) * N,
          min(wrap(side ? k0 + TK : k0 - 1), N - 1));
  }
  __syncthreads();

  // phase 2: two cells of a row in kPlanes planes a thread
  const int t2 = threadIdx.x % (kThreads / 2), half = threadIdx.x / (kThreads / 2);
  const int tk = t2 % (TK / 2) * 2, tj = t2 / (TK / 2);
  const int gj = j0 + tj, gk = k0 + tk, i1 = i0 + half * kPlanes;
  if (gj >= N || gk >= N || i1 >= N) return;
  const bool whole = PAIR || gk + 1 < N;
  const int at = (half * kPlanes * HJ + tj + 1) * HK + 2 + tk;  // plane i1 - 1
  const auto load = [&](const float* p) {
    if constexpr (PAIR) {
      const float2 v = __ldg(reinterpret_cast<const float2*>(p));
      return pk(v.x, v.y);
    } else {
      return pk(__ldg(p), whole ? __ldg(p + 1) : 0.0f);
    }
  };
  const auto store = [&](float* p, float x, float y) {
    if constexpr (PAIR) {
      *reinterpret_cast<float2*>(p) = make_float2(x, y);
    } else {
      p[0] = x;
      if (whole) p[1] = y;
    }
  };
  F2 lapR[kPlanes], ur[kPlanes], lapX[kPlanes], gx[kPlanes];
  F2 lapI[kPlanes], ui[kPlanes], Pr[kPlanes], Pi[kPlanes], dPr[kPlanes], dPi[kPlanes],
      dwPr[kPlanes], dwPi[kPlanes], unused[kPlanes];
  lap_pairs(S.f[0], at, lapR, ur);
  lap_pairs(S.f[1], at, lapX, gx);
  if constexpr (LEVEL == LFM_COMPLEX) {
    lap_pairs(S.f[2], at, lapI, ui);
    dsum_pairs(S.f[3], at, dPr, Pr);
    dsum_pairs(S.f[4], at, dPi, Pi);
    dsum_pairs(S.f[5], at, dwPr, unused);
    dsum_pairs(S.f[6], at, dwPi, unused);
  }
  const int qjk[2] = {qterm(gj, N) + qterm(gk, N), qterm(gj, N) + qterm(whole ? gk + 1 : gk, N)};
#pragma unroll
  for (int p = 0; p < kPlanes; ++p) {
    const int gi = i1 + p;
    if (gi >= N) break;
    const int64_t x = ((int64_t)gi * N + gj) * N + gk;
    const int qi = qterm(gi, N);
    const F2 X_ = load(A.chi + x), prp = load(A.g_prp + x), chip = load(A.g_chip + x);
    F2 pip, E_;
    if constexpr (LEVEL == LFM_COMPLEX)
      pip = load(A.g_pip + x);
    else
      E_ = load(A.pr + x);
    float o_pr[2], o_pi[2], o_chi[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const auto of = [e](const F2& v) { return e ? v.v.y : v.v.x; };
      const float m0 = mask_from_q_flat(A.lut, qi + qjk[e]), a0 = fsub(1.0f, m0);
      const float X = of(X_), X2 = X * X, u = of(ur[p]), g = of(gx[p]);
      const float gacc = A.dt2 * g;
      const float gQ = -gacc * A.K * X;
      const float hp = A.use_lambda ? A.four_lambda * (3.0f * X2 - A.chi0_sq) : 0.0f;
      if constexpr (LEVEL == LFM_COMPLEX) {
        const float v = of(ui[p]), R = of(Pr[p]), I = of(Pi[p]);
        const float dR = of(dPr[p]), dI = of(dPi[p]);
        const float jt = 0.5f * (R * dI - I * dR);
        const float Q = R * R + I * I + A.eps_w * jt - A.e0_sq;
        const float w0 = 0.5f * A.eps_w * gQ;
        o_pr[e] = a0 * of(prp) + 2.0f * u + A.dt2 * of(lapR[p]) - A.dt2 * X2 * u +
                  2.0f * R * gQ + w0 * dI + of(dwPi[p]);
        o_pi[e] = a0 * of(pip) + 2.0f * v + A.dt2 * of(lapI[p]) - A.dt2 * X2 * v +
                  2.0f * I * gQ - w0 * dR - of(dwPr[p]);
        o_chi[e] = of(chip) + 2.0f * g + A.dt2 * of(lapX[p]) - gacc * (hp + A.K * Q) -
                   2.0f * A.dt2 * X * (R * u + I * v);
      } else {
        const float E = of(E_);
        const float Q = E * E - A.e0_sq;
        o_pr[e] = a0 * of(prp) + 2.0f * u + A.dt2 * of(lapR[p]) - A.dt2 * X2 * u + 2.0f * E * gQ;
        o_chi[e] = of(chip) + 2.0f * g + A.dt2 * of(lapX[p]) - gacc * (hp + A.K * Q) -
                   2.0f * A.dt2 * X * E * u;
      }
      if constexpr (U_OUT) {  // chi is the chi_next of the step before
        o_pr[e] = a0 * o_pr[e];
        if constexpr (LEVEL == LFM_COMPLEX) o_pi[e] = a0 * o_pi[e];
        o_chi[e] = X != clamp_value(A, m0, a0) ? a0 * o_chi[e] : 0.0f;
      }
    }
    store(A.o_pr + x, o_pr[0], o_pr[1]);
    store(A.o_prp + x, -ur[p].v.x, -ur[p].v.y);
    store(A.o_chi + x, o_chi[0], o_chi[1]);
    store(A.o_chip + x, -gx[p].v.x, -gx[p].v.y);
    if constexpr (LEVEL == LFM_COMPLEX) {
      store(A.o_pi + x, o_pi[0], o_pi[1]);
      store(A.o_pip + x, -ui[p].v.x, -ui[p].v.y);
    }
  }
}

template <int LEVEL, bool PAIR, bool U_IN, bool U_OUT>
cudaError_t launch(const AdjArgs& A, int tiles, cudaStream_t stream) {
  const int smem = (int)sizeof(TileSmem<LEVEL>);
  const auto kernel = adjoint_tile_kernel<LEVEL, PAIR, U_IN, U_OUT>;
  if (smem > 48 * 1024) {  // above the default: granted per device, not once a process
    cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  kernel<<<tiles, kThreads, smem, stream>>>(A);
  return cudaGetLastError();
}

template <int LEVEL, bool PAIR>
cudaError_t launch_chain(const AdjArgs& A, int chain, int tiles, cudaStream_t stream) {
  switch (chain) {
    case 0: return launch<LEVEL, PAIR, false, false>(A, tiles, stream);
    case 1: return launch<LEVEL, PAIR, true, false>(A, tiles, stream);
    case 2: return launch<LEVEL, PAIR, false, true>(A, tiles, stream);
    default: return launch<LEVEL, PAIR, true, true>(A, tiles, stream);
  }
}

}  // namespace

cudaError_t launch_adjoint_step(int level, int N, const float* pr, const float* pi,
                                const float* chi, const float* chi_next, const MaskLut& lut,
                                const float* const g_out[6], float* const g_in[6],
                                const StepConsts& c, int chain, cudaStream_t stream) {
  AdjArgs A{};
  A.level = level;
  A.N = N;
  A.pr = pr;
  A.pi = pi;
  A.chi = chi;
  A.chi_next = chi_next;
  A.lut = lut;
  A.g_pr = g_out[0]; A.g_prp = g_out[1]; A.g_pi = g_out[2]; A.g_pip = g_out[3];
  A.g_chi = g_out[4]; A.g_chip = g_out[5];
  A.o_pr = g_in[0]; A.o_prp = g_in[1]; A.o_pi = g_in[2]; A.o_pip = g_in[3];
  A.o_chi = g_in[4]; A.o_chip = g_in[5];
  A.dt2 = c.dt2;
  A.K = c.k_over_chi0;
  A.eps_w = c.eps_w;
  A.e0_sq = c.e0_sq;
  A.four_lambda = c.four_lambda;
  A.chi0 = c.chi0;
  A.chi0_sq = c.chi0_sq;
  A.neg_chi0 = c.neg_chi0;
  A.use_lambda = c.use_lambda;
  const int tiles = ((N + TK - 1) / TK) * ((N + TJ - 1) / TJ) * ((N + TI - 1) / TI);
  bool pair = N % 2 == 0;
  for (const void* p : {(const void*)pr, (const void*)chi, (const void*)A.g_prp,
                        (const void*)A.g_pip, (const void*)A.g_chip, (const void*)A.o_pr,
                        (const void*)A.o_prp, (const void*)A.o_pi, (const void*)A.o_pip,
                        (const void*)A.o_chi, (const void*)A.o_chip})
    pair = pair && (reinterpret_cast<uintptr_t>(p) & 7u) == 0;
  if (level == LFM_REAL)
    return pair ? launch_chain<LFM_REAL, true>(A, chain, tiles, stream)
                : launch_chain<LFM_REAL, false>(A, chain, tiles, stream);
  return pair ? launch_chain<LFM_COMPLEX, true>(A, chain, tiles, stream)
              : launch_chain<LFM_COMPLEX, false>(A, chain, tiles, stream);
}

}  // namespace lfm
