// Marching step kernels through L1, for lattices the copy engine cannot serve and
// those it serves more slowly.
//
// The fused kernels of step_tma.cu copy rows in 16-byte units, so they need N % 4
// == 0 and aligned fields.  Here a thread keeps two cells of a row and marches along
// i with the register queue of the fused kernels, four planes deep: a plane's values
// are loaded through L1 once, a plane before they are needed, and serve as next,
// centre and previous plane.  A CTA owns a run of consecutive threads of the (j, k)
// plane, several rows long, so most neighbouring rows are its own.
//
// Against the direct kernel (a thread per cell, 38 loads and a 64-bit index each at
// REAL), us a step: REAL 110^3 28.0 -> 15.3, 125^3 38.2 -> 20.8, 150^3 62.5 -> 29.0,
// 250^3 288 -> 145, 333^3 673 -> 306; COMPLEX 127^3 52.6 -> 36.2, 150^3 90.4 -> 51.7,
// 250^3 415 -> 228; split chi 150^3 69.9 -> 43.1.  12 to 16 warps an SM (the queue's
// registers) leave it waiting for loads: one cell a thread without the load ahead gave
// odd edges nothing at 333^3 (687), two cells give them 306.
//
// Arithmetic: lfm_cells.cuh in the order of the other kernels, bit-identical.
#include <algorithm>
#include <type_traits>

#include "lfm_kernels.h"
#include "lfm_queue.cuh"

namespace lfm {
namespace {

constexpr int kPlain = 0, kComp = 1, kSplit = 2;
constexpr int V = 2;  // cells a thread

template <int LEVEL>
constexpr int kFields = LEVEL == LFM_REAL ? 2 : 3;
// Two CTAs an SM, with the registers a queue of four planes takes.
template <int LEVEL>
constexpr int kThreads = LEVEL == LFM_REAL ? 256 : 192;

// A thread's rows in a plane, as offsets from the plane's start, and its neighbours
// in k as offsets from its first cell: the one before, its second cell (the row's
// first cell when the row ends at the first: N odd) and the one after.
struct Rows {
  int m, z, p, left, two, right;
  bool whole;  // both cells lie in the row
};

__device__ __forceinline__ Rows rows_at(int N, int j, int k0) {
  Rows R;
  R.z = j * N + k0;
  R.m = (j == 0 ? N - 1 : j - 1) * N + k0;
  R.p = (j == N - 1 ? 0 : j + 1) * N + k0;
  R.whole = k0 + 1 < N;
  R.left = k0 == 0 ? N - 1 : -1;
  R.two = R.whole ? 1 : -k0;
  R.right = k0 + V < N ? V : (k0 + V == N ? -k0 : 0);
  return R;
}

// The two cells at p; PAIR: as one 8-byte load (N even, aligned fields).
template <bool PAIR>
__device__ __forceinline__ Vec<V> ldg2(const float* p, const Rows& R) {
  Vec<V> r;
  if constexpr (PAIR) {
    const float2 t = __ldg(reinterpret_cast<const float2*>(p));
    r.v[0] = t.x; r.v[1] = t.y;
  } else {
    r.v[0] = __ldg(p);
    r.v[1] = __ldg(p + R.two);
  }
  return r;
}

// The cells' own values of a field that this launch may overwrite there (no
// read-only path).
template <bool PAIR>
__device__ __forceinline__ Vec<V> own2(const float* p, const Rows& R) {
  Vec<V> r;
  if constexpr (PAIR) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    r.v[0] = t.x; r.v[1] = t.y;
  } else {
    r.v[0] = *p;
    r.v[1] = R.whole ? p[1] : 0.0f;
  }
  return r;
}

template <bool PAIR>
__device__ __forceinline__ void put2(float* p, const float (&x)[V], const Rows& R) {
  if constexpr (PAIR) {
    stg<V>(p, x);
  } else {
    p[0] = x[0];
    if (R.whole) p[1] = x[1];
  }
}

template <bool PAIR>
__device__ __forceinline__ void load_plane(QPlane<V>& q, const float* f, const Rows& R) {
  q.m = ldg2<PAIR>(f + R.m, R);
  q.z = ldg2<PAIR>(f + R.z, R);
  q.p = ldg2<PAIR>(f + R.p, R);
  q.zl = __ldg(f + R.z + R.left);
  q.zr = __ldg(f + R.z + R.right);
}

__device__ __forceinline__ void load_sides(QPlane<V>& q, const float* f, const Rows& R) {
  q.ml = __ldg(f + R.m + R.left);
  q.mr = __ldg(f + R.m + R.right);
  q.pl = __ldg(f + R.p + R.left);
  q.pr = __ldg(f + R.p + R.right);
}

// The cells' own values of a plane: previous fields, chi's (split) lo parts, and the
// streamed mask or none.
struct Points {
  Vec<V> r, i, c, lo, lo_prev, mask;
};

template <int LEVEL, int MODE, bool PAIR>
__device__ __forceinline__ void load_points(Points& p, const StepArgs& a, int64_t x,
                                            const Rows& R) {
  p.r = own2<PAIR>(a.pr_prev + x, R);
  p.c = own2<PAIR>(a.chi_prev + x, R);
  if constexpr (LEVEL == LFM_COMPLEX) p.i = own2<PAIR>(a.pi_prev + x, R);
  if constexpr (MODE == kSplit) {
    p.lo = own2<PAIR>(a.chi_lo + x, R);
    p.lo_prev = own2<PAIR>(a.chi_lo_prev + x, R);
  }
  if (a.mask) p.mask = own2<PAIR>(a.mask + x, R);
}

// One plane of a thread's march: updates the cells of plane i (its queue slots PA,
// PB, PC; `here` its start in a field) and loads plane i+2 into slot PD (`ahead`) and
// the points of plane i+1 (`after`), so that a plane's loads have the plane before to
// arrive in.
template <int LEVEL, int MODE, bool PAIR, int PA, int PB, int PC, int PD>
__device__ __forceinline__ void plane(const StepArgs& a, QPlane<V> (&Q)[kFields<LEVEL>][4],
                                      Points& pts, const Rows& R, const int32_t (&qjk)[V], int i,
                                      int64_t here, int64_t after, int64_t ahead, bool more) {
  constexpr int NS = kFields<LEVEL>;
  const float* f[3] = {a.pr, LEVEL == LFM_REAL ? a.chi : a.pi, a.chi};
  const Points now = pts;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    load_sides(Q[s][PB], f[s] + here, R);
    if (more) load_plane<PAIR>(Q[s][PD], f[s] + ahead, R);
  }
  if (more) load_points<LEVEL, MODE, PAIR>(pts, a, after + R.z, R);
  const int64_t x = here + R.z;
  float mask[V], absorb[V];
  if (a.mask) {
#pragma unroll
    for (int e = 0; e < V; ++e) mask[e] = now.mask.v[e];
  } else {
    const int32_t qi = qterm(i + a.i_off, a.N);
#pragma unroll
    for (int e = 0; e < V; ++e) mask[e] = mask_from_q_flat(a.lut, qi + qjk[e]);
  }
#pragma unroll
  for (int e = 0; e < V; ++e) absorb[e] = fsub(1.0f, mask[e]);
  const Vec<V>&rp = now.r, &ip = now.i, &cp = now.c;
  float o_r[V], o_i[V], o_c[V], o_rp[V], o_ip[V], o_cp[V];
  constexpr int C = NS - 1;  // chi's queue
  if constexpr (MODE == kSplit) {
    const Vec<V>&lc = now.lo, &lp = now.lo_prev;
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const S19 R0 = q_s19<V>(Q[0][PA], Q[0][PB], Q[0][PC], e);
      const S19 H = q_s19<V>(Q[C][PA], Q[C][PB], Q[C][PC], e);
      const double d = split_value(H.c, lc.v[e]), dp = split_value(cp.v[e], lp.v[e]);
      const float rpv = a.damp_prev ? fmul(rp.v[e], absorb[e]) : rp.v[e];
      SplitChi chi;
      if constexpr (LEVEL == LFM_REAL) {
        const RealSplit o = real_cell_split(lap19_fma(R0), R0.c, rpv, lap19_diff(H), d, dp,
                                            mask[e], absorb[e], a.c);
        o_r[e] = o.psi;
        chi = o.chi;
      } else {
        const S19 I0 = q_s19<V>(Q[1][PA], Q[1][PB], Q[1][PC], e);
        const float ipv = a.damp_prev ? fmul(ip.v[e], absorb[e]) : ip.v[e];
        const ComplexSplit o =
            complex_cell_split(lap19_fma(R0), R0.c, rpv, faces_of(R0), lap19_fma(I0), I0.c, ipv,
                               faces_of(I0), lap19_diff(H), d, dp, mask[e], absorb[e], a.c);
        o_r[e] = o.pr;
        o_i[e] = o.pi;
        chi = o.chi;
      }
      o_c[e] = chi.hi;
      o_cp[e] = chi.lo;
    }
    put2<PAIR>(a.pr_out + x, o_r, R);
    if constexpr (LEVEL == LFM_COMPLEX) put2<PAIR>(a.pi_out + x, o_i, R);
    put2<PAIR>(a.chi_out + x, o_c, R);
    put2<PAIR>(a.chi_lo_out + x, o_cp, R);
    return;
  } else if constexpr (MODE == kComp) {
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const S19 R0 = q_s19<V>(Q[0][PA], Q[0][PB], Q[0][PC], e);
      const S19 X = q_s19<V>(Q[C][PA], Q[C][PB], Q[C][PC], e);
      if constexpr (LEVEL == LFM_REAL) {
        const RealComp o = real_cell_comp(lap19_fma(R0), R0.c, rp.v[e], lap19_diff(X), X.c,
                                          cp.v[e], mask[e], a.c);
        o_r[e] = o.psi.v; o_rp[e] = o.psi.d; o_c[e] = o.chi.v; o_cp[e] = o.chi.d;
      } else {
        const S19 I0 = q_s19<V>(Q[1][PA], Q[1][PB], Q[1][PC], e);
        const ComplexComp o = complex_cell_comp(lap19_fma(R0), R0.c, rp.v[e], faces_of(R0),
                                                lap19_fma(I0), I0.c, ip.v[e], faces_of(I0),
                                                lap19_diff(X), X.c, cp.v[e], mask[e], a.c);
        o_r[e] = o.pr.v; o_rp[e] = o.pr.d; o_i[e] = o.pi.v; o_ip[e] = o.pi.d;
        o_c[e] = o.chi.v; o_cp[e] = o.chi.d;
      }
    }
  } else {
    S19 R0[V], I0[V], X[V];
#pragma unroll
    for (int e = 0; e < V; ++e) {
      R0[e] = q_s19<V>(Q[0][PA], Q[0][PB], Q[0][PC], e);
      X[e] = q_s19<V>(Q[C][PA], Q[C][PB], Q[C][PC], e);
      if constexpr (LEVEL == LFM_COMPLEX) I0[e] = q_s19<V>(Q[1][PA], Q[1][PB], Q[1][PC], e);
    }
    const auto pair = [](const auto& v) { return pk(v[0], v[1]); };
    const auto put = [](float (&o)[V], const F2& t) { o[0] = t.v.x; o[1] = t.v.y; };
    const auto centre = [](const S19 (&s)[V]) { return pk(s[0].c, s[1].c); };
    const auto faces = [](const S19 (&s)[V]) { return pk_faces(faces_of(s[0]), faces_of(s[1])); };
    const F2 mk = pair(mask), ab = fsub(cst<F2>(1.0f), mk);
    F2 rpv = pair(rp.v);
    if (a.damp_prev) rpv = fmul(rpv, ab);
    if constexpr (LEVEL == LFM_REAL) {
      const RealOutT<F2> o = real_cell_ab(lap19_pair(R0[0], R0[1]), centre(R0), rpv,
                                          lap19_pair(X[0], X[1]), centre(X), pair(cp.v), mk, ab,
                                          a.c);
      put(o_r, o.psi); put(o_rp, o.psi_prev); put(o_c, o.chi); put(o_cp, o.chi_prev);
    } else {
      F2 ipv = pair(ip.v);
      if (a.damp_prev) ipv = fmul(ipv, ab);
      const ComplexOutT<F2> o = complex_cell_ab(
          lap19_pair(R0[0], R0[1]), centre(R0), rpv, faces(R0), lap19_pair(I0[0], I0[1]),
          centre(I0), ipv, faces(I0), lap19_pair(X[0], X[1]), centre(X), pair(cp.v), mk, ab, a.c);
      put(o_r, o.pr); put(o_rp, o.pr_prev); put(o_i, o.pi); put(o_ip, o.pi_prev);
      put(o_c, o.chi); put(o_cp, o.chi_prev);
    }
  }
  put2<PAIR>(a.pr_out + x, o_r, R);
  put2<PAIR>(a.chi_out + x, o_c, R);
  if (a.pr_prev_out) put2<PAIR>(a.pr_prev_out + x, o_rp, R);
  if (a.chi_prev_out) put2<PAIR>(a.chi_prev_out + x, o_cp, R);
  if constexpr (LEVEL == LFM_COMPLEX) {
    put2<PAIR>(a.pi_out + x, o_i, R);
    if (a.pi_prev_out) put2<PAIR>(a.pi_prev_out + x, o_ip, R);
  }
}

template <int LEVEL, int MODE, bool PAIR>
__global__ void __launch_bounds__(kThreads<LEVEL>, 2)
    march_step_kernel(const __grid_constant__ StepArgs a, int planes, int tiles) {
  constexpr int NS = kFields<LEVEL>;
  const int N = a.N, groups = (N + 1) / V, n2 = N * N;
  const int y = (blockIdx.x % tiles) * kThreads<LEVEL> + threadIdx.x;
  if (y >= N * groups) return;
  const int j = y / groups, k0 = (y - j * groups) * V;
  const Rows R = rows_at(N, j, k0);
  int32_t qjk[V];
#pragma unroll
  for (int e = 0; e < V; ++e) qjk[e] = qterm(j, N) + qterm(min(k0 + e, N - 1), N);
  const int lo = a.slab ? a.i_lo : 0, hi = a.slab ? a.i_hi : N;
  const int i0 = lo + (int)(blockIdx.x / tiles) * planes, i1 = min(i0 + planes, hi);
  // a slab reads its ghost planes, a whole lattice wraps
  const auto at = [&](int i) {
    const int w = a.slab ? i : (i < 0 ? i + N : (i >= N ? i - N : i));
    return (int64_t)w * n2;
  };
  QPlane<V> Q[NS][4];
  Points pts;
  const float* f[3] = {a.pr, LEVEL == LFM_REAL ? a.chi : a.pi, a.chi};
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    load_plane<PAIR>(Q[s][0], f[s] + at(i0 - 1), R);
    load_plane<PAIR>(Q[s][1], f[s] + at(i0), R);
    load_plane<PAIR>(Q[s][2], f[s] + at(i0 + 1), R);
  }
  load_points<LEVEL, MODE, PAIR>(pts, a, at(i0) + R.z, R);
  for (int i = i0; i < i1;) {
#define LFM_MARCH(A, B, C, D)                                                             \
  plane<LEVEL, MODE, PAIR, A, B, C, D>(a, Q, pts, R, qjk, i, at(i), at(i + 1), at(i + 2), \
                                       i + 1 < i1);                                       \
  if (++i >= i1) break;
    LFM_MARCH(0, 1, 2, 3)
    LFM_MARCH(1, 2, 3, 0)
    LFM_MARCH(2, 3, 0, 1)
    LFM_MARCH(3, 0, 1, 2)
#undef LFM_MARCH
  }
}

// ---- COLOR ------------------------------------------------------------------
// Seven stencil fields do not fit into a register queue, so a plane's three planes of
// rows are loaded for each field in turn; marching along i, a CTA finds two of the
// three in L1.  Two cells a thread run packed, as in the fused kernel.  Without S_a, us
// a step, against the direct kernel: 50^3 11.4 -> 8.4, 110^3 97.9 -> 68.3, 150^3 256 ->
// 178, 210^3 711 -> 458; against the fused kernel's run-time tile: 72^3 26.3 -> 19.7,
// 144^3 164 -> 141, 160^3 210 -> 193, 288^3 1272 -> 1093 (the tile where it has warps
// enough: run_time_tile_pays in step_tma.cu).
template <bool PAIR>
__global__ void __launch_bounds__(256, 2)
    march_color_kernel(const __grid_constant__ StepArgs a, int planes, int tiles) {
  const int N = a.N, groups = (N + 1) / V, n2 = N * N;
  const int y = (blockIdx.x % tiles) * 256 + threadIdx.x;
  if (y >= N * groups) return;
  const int j = y / groups, k0 = (y - j * groups) * V;
  const Rows R = rows_at(N, j, k0);
  const int64_t n3 = (int64_t)n2 * N;
  const int32_t qj0 = qterm(j, N) + qterm(k0, N), qj1 = qterm(j, N) + qterm(min(k0 + 1, N - 1), N);
  const int i0 = (int)(blockIdx.x / tiles) * planes, i1 = min(i0 + planes, N);
  const auto pair = [](const Vec<V>& v) { return pk(v.v[0], v.v[1]); };
  const auto put = [&](float* p, const F2& t) {
    const float o[V] = {t.v.x, t.v.y};
    put2<PAIR>(p, o, R);
  };
  for (int i = i0; i < i1; ++i) {
    const int64_t here = (int64_t)i * n2, x = here + R.z;
    const int64_t before = (int64_t)(i == 0 ? N - 1 : i - 1) * n2;
    const int64_t after = (int64_t)(i == N - 1 ? 0 : i + 1) * n2;
    // the Laplacian, centre and faces of field f at the thread's cells
    S19 c0, c1;
    const auto gather = [&](const float* f) {
      QPlane<V> m, c, p;
      load_plane<PAIR>(m, f + before, R);
      load_plane<PAIR>(c, f + here, R);
      load_sides(c, f + here, R);
      load_plane<PAIR>(p, f + after, R);
      c0 = q_s19<V>(m, c, p, 0);
      c1 = q_s19<V>(m, c, p, 1);
    };
    F2 mask;
    if (a.mask) {
      mask = pair(own2<PAIR>(a.mask + x, R));
    } else {
      const int32_t qi = qterm(i, N);
      mask = pk(mask_from_q_flat(a.lut, qi + qj0), mask_from_q_flat(a.lut, qi + qj1));
    }
    F2 prc[3], pic[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      prc[c] = pair(ldg2<PAIR>(a.pr + c * n3 + x, R));
      pic[c] = pair(ldg2<PAIR>(a.pi + c * n3 + x, R));
    }
    gather(a.chi);
    const F2 lapX = lap19_pair(c0, c1), chi = pk(c0.c, c1.c);
    ColorAccT<F2> A;
    color_begin(A, chi, mask, prc, pic, a.c);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      F2 rp = pair(own2<PAIR>(a.pr_prev + c * n3 + x, R));
      F2 ip = pair(own2<PAIR>(a.pi_prev + c * n3 + x, R));
      if (a.damp_prev) {
        rp = fmul(rp, A.absorb);
        ip = fmul(ip, A.absorb);
      }
      gather(a.pr + c * n3);
      const F2 lapR = lap19_pair(c0, c1), pr = pk(c0.c, c1.c);
      const FacesT<F2> fr = pk_faces(faces_of(c0), faces_of(c1));
      gather(a.pi + c * n3);
      const ColorCompOutT<F2> o =
          color_component(A, c, lapR, pr, rp, fr, lap19_pair(c0, c1), pk(c0.c, c1.c), ip,
                          pk_faces(faces_of(c0), faces_of(c1)), a.c);
      put(a.pr_out + c * n3 + x, o.pr);
      put(a.pi_out + c * n3 + x, o.pi);
      if (a.energy_out)
        put(a.energy_out + c * n3 + x, fadd(fmul(o.pr, o.pr), fmul(o.pi, o.pi)));
      if (a.pr_prev_out) put(a.pr_prev_out + c * n3 + x, o.pr_prev);
      if (a.pi_prev_out) put(a.pi_prev_out + c * n3 + x, o.pi_prev);
    }
    F2 sa[3] = {cst<F2>(0.0f), cst<F2>(0.0f), cst<F2>(0.0f)};
    if (a.sa) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        sa[c] = pair(ldg2<PAIR>(a.sa + c * n3 + x, R));
        if (a.sa_clip_out)
          put(a.sa_clip_out + c * n3 + x, pk(fmaxf(sa[c].v.x, 0.0f), fmaxf(sa[c].v.y, 0.0f)));
      }
    }
    const F2 xp = pair(own2<PAIR>(a.chi_prev + x, R));
    put(a.chi_out + x, color_finish(A, lapX, xp, a.sa != nullptr, sa, a.c));
    if (a.chi_prev_out) put(a.chi_prev_out + x, chi);
  }
}

int color_tiles(int N) { return (N * ((N + 1) / V) + 255) / 256; }

cudaError_t launch_color(const StepArgs& a, bool pairs, cudaStream_t stream) {
  const int tiles = color_tiles(a.N);
  const int64_t work = (int64_t)tiles * a.N;
  // All CTAs resident at once (2 x 148) while that takes ten planes or fewer (110^3: 68.3
  // us with nine, 78 with four, 74 with one), four planes beyond (150^3: 178 with four,
  // 188 with one, 223 with 16).
  int planes = (int)((work + 295) / 296);
  if (planes > 10) planes = 4;
  const unsigned grid = (unsigned)tiles * (unsigned)((a.N + planes - 1) / planes);
  if (pairs)
    march_color_kernel<true><<<grid, 256, 0, stream>>>(a, planes, tiles);
  else
    march_color_kernel<false><<<grid, 256, 0, stream>>>(a, planes, tiles);
  return cudaGetLastError();
}

template <int LEVEL, int MODE>
cudaError_t launch(const StepArgs& a, bool pairs, cudaStream_t stream) {
  const int threads = kThreads<LEVEL>, range = a.slab ? a.i_hi - a.i_lo : a.N;
  const int tiles = (a.N * ((a.N + 1) / V) + threads - 1) / threads;
  // Planes a march.  A small lattice takes as few as keep all CTAs resident (2 x 148;
  // REAL 46^3: 4.2 us with 1 plane, 6.3 with 4).  Beyond four planes that way, long
  // marches amortise their two extra planes, with four CTAs or more a resident slot
  // so that the last wave is short: within 5 % of the best of 4, 8, 16, 24 and 32
  // planes at the sizes above but REAL 250^3 (8 %).
  const int64_t work = (int64_t)tiles * range;
  int planes = (int)((work + 295) / 296);
  if (planes > 4) planes = (int)std::min<int64_t>(32, std::max<int64_t>(4, work / (4 * 296)));
  planes = std::min(planes, range);
  const unsigned grid = (unsigned)tiles * (unsigned)((range + planes - 1) / planes);
  if (pairs)
    march_step_kernel<LEVEL, MODE, true><<<grid, threads, 0, stream>>>(a, planes, tiles);
  else
    march_step_kernel<LEVEL, MODE, false><<<grid, threads, 0, stream>>>(a, planes, tiles);
  return cudaGetLastError();
}

// Whether the march beats the direct kernel, whose one-cell threads are done sooner on the
// smallest lattices.  us a step, march / direct (every edge from 32 to 65 measured):
//
// - REAL: from 32^3 (32^3 2.53 / 2.64, 33^3 2.51 / 2.86, 48^3 3.39 / 4.05; 30^3 4.2 / 3.2),
//   COMPLEX from 32^3 by pairs (34^3 3.42 / 3.76, 46^3 3.92 / 4.87) and, compensated,
//   without (33^3 3.51 / 3.53, 37^3 3.50 / 4.03).
// - Without pairs COMPLEX, and REAL compensated and split chi, from 43^3: COMPLEX 33^3
//   3.96 / 3.32, 41^3 4.51 / 3.94, 43^3 4.51 / 4.74; split REAL 41^3 3.84 / 3.50, 43^3
//   3.82 / 4.15.
// - COLOR from 45^3 (9.27 / 10.2; 44^3 9.99 / 9.98) to the edge whose planes no longer find
//   room at once (50^3 8.38 / 11.4; 51^3 15.1 / 11.7, 53^3 15.3 / 11.9) and from 54^3 (13.4 /
//   14.1), without pairs 59^3 (15.8 / 16.4; 57^3 15.7 / 15.1), on.
bool marching_pays(const StepArgs& a, bool pairs) {
  if (a.level == LFM_COLOR)
    return !a.slab && a.N >= 45 &&
           (a.N >= (pairs ? 54 : 59) || color_tiles(a.N) * a.N <= 2 * 148);
  const bool from_32 = pairs || (a.level == LFM_REAL ? !a.comp && !a.split : a.comp != 0);
  return a.N >= (from_32 ? 32 : 43);
}

}  // namespace

cudaError_t launch_march_step(const StepArgs& a, cudaStream_t stream) {
  // two cells a thread where every row starts on 8 bytes
  bool pairs = a.N % 2 == 0;
  const void* ptrs[] = {a.pr, a.pi, a.chi, a.pr_prev, a.pi_prev, a.chi_prev, a.pr_out, a.pi_out,
                        a.chi_out, a.pr_prev_out, a.pi_prev_out, a.chi_prev_out, a.mask,
                        a.chi_lo, a.chi_lo_prev, a.chi_lo_out, a.sa, a.sa_clip_out,
                        a.energy_out};
  for (const void* p : ptrs) pairs = pairs && (reinterpret_cast<uintptr_t>(p) & 7u) == 0;
  if (!marching_pays(a, pairs)) return cudaErrorNotSupported;
  if (a.level == LFM_COLOR) return launch_color(a, pairs, stream);
  if (a.level == LFM_REAL)
    return a.split  ? launch<LFM_REAL, kSplit>(a, pairs, stream)
           : a.comp ? launch<LFM_REAL, kComp>(a, pairs, stream)
                    : launch<LFM_REAL, kPlain>(a, pairs, stream);
  return a.split  ? launch<LFM_COMPLEX, kSplit>(a, pairs, stream)
         : a.comp ? launch<LFM_COMPLEX, kComp>(a, pairs, stream)
                  : launch<LFM_COMPLEX, kPlain>(a, pairs, stream);
}

}  // namespace lfm
