// Many leapfrog steps of a small lattice in one launch, the state held on chip.
//
// A lattice of up to about 100^3 cells fits into the SMs' shared memory
// (148 x 227 KB).  The step kernels of step_tma.cu read and write all of it
// every step and are launched once a step; at these sizes a step is then all
// latency: launch, pipeline fill, one pass through L2.  Here one cooperative
// launch runs all steps.  Every CTA (one per SM) owns a block of ni x nj whole
// k rows, keeps both time levels of it in shared memory, and per step exchanges
// only the rows that border its neighbours, through L2.
//
// A step marches the block's planes along i (register queue, as step_tma.cu).  A
// new value goes over the previous one in shared memory.  The cells of an outer
// row go to an exchange buffer as well, in 16-byte packets of three values and
// the number of their time level, each written and read as one 128-bit memory
// operation.  A reader polls the packets themselves until they carry the time
// level it needs: one store and one load of latency, where a flag behind a fence
// took a fence, a flag's round trip and the data's (measured at REAL 32^3: 1230 +
// 1470 + 3550 cycles of a step's 7500).
//
// Two buffers, by the parity of the time level, are enough: packets of time t go
// over those of time t-2, and a block writes them only after it has read all
// neighbours' packets of time t-1, which a neighbour writes after its last read
// of time t-2.  Time levels are counted on from a base that the last CTA to
// retire moves on, so a workspace serves launch after launch without being
// cleared.  The field slots in global memory are read at the start and written
// with the last two time levels, as the per-step kernels leave them.
//
// Arithmetic: lfm_cells.cuh in the order of the other kernels, bit-identical.
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "lfm_kernels.h"
#include "lfm_launch.h"
#include "lfm_queue.cuh"
#include "lfm_resident.h"

namespace lfm {
namespace {

constexpr int kMaxThreads = 512;
constexpr int kThreadsComplex = 384;  // COMPLEX takes up to 168 registers
constexpr int kMaxBlocks = 148;  // one block an SM
// Cells a thread: two (one packed pair).  Four were slower at every REAL size (64^3
// 3.99 against 3.53 us a step, 96^3 8.1 against 7.5): their k neighbours meet in
// four-way bank conflicts, and half the threads are left to hide latency.
constexpr int kCells = 2;
constexpr int kSmallEdge = 36;
constexpr int kSmemBytes = 226 * 1024;  // 227 KB opt-in less the static part

template <int LEVEL>
constexpr int kFields = LEVEL == LFM_REAL ? 2 : 3;

// 16-byte packets a group of V cells takes: three values and the time level each.
template <int LEVEL, int V>
constexpr int kPackets = (kFields<LEVEL> * V + 2) / 3;

struct Packet {
  float v[3];
  uint32_t t;
};

// A packet is read and written as one: .b128 is a scalar type to PTX (sm_70 on), and its
// memory model takes a strong operation on a scalar as one operation on all the bytes
// (one on a vector, as ld.v4.b32, as an operation for each element, in any order).  The
// 16-byte atomic loads and stores of CUDA C++ (__nv_atomic_load, __nv_atomic_store) rest on
// the same access; written with them the kernel took 6 % less (REAL 33^3) to 4 % more time
// (COMPLEX 36^3), 1 % more at REAL 32^3.
__device__ __forceinline__ void st_packet(ulonglong2* p, const Packet& x) {
  unsigned long long lo, hi;
  memcpy(&lo, &x.v[0], 8);
  memcpy(&hi, &x.v[2], 8);
  asm volatile(
      "{\n\t.reg .b128 d;\n\t"
      "mov.b128 d, {%1, %2};\n\t"
      "st.relaxed.gpu.global.b128 [%0], d;\n\t}" ::"l"(p), "l"(lo), "l"(hi)
      : "memory");
}

__device__ __forceinline__ Packet ld_packet(const ulonglong2* p) {
  unsigned long long lo, hi;
  asm volatile(
      "{\n\t.reg .b128 d;\n\t"
      "ld.relaxed.gpu.global.b128 d, [%2];\n\t"
      "mov.b128 {%0, %1}, d;\n\t}"
      : "=l"(lo), "=l"(hi)
      : "l"(p)
      : "memory");
  Packet x;
  memcpy(&x.v[0], &lo, 8);
  memcpy(&x.v[2], &hi, 8);
  return x;
}

// Whether a packet of VALUES values carries time level t.  Its spare places carry
// the level as well and are looked at too, so that every word of the load is used: with
// spare words left unused (REAL, two cells a thread) packets were seen whose words did
// not belong together.  The cause was not found; a load made narrower in compilation,
// where a part of its result is not used, would explain it.  The packets without spare
// words use all of theirs.
template <int VALUES>
__device__ __forceinline__ bool carries(const Packet& x, uint32_t t) {
  bool ok = x.t == t;
#pragma unroll
  for (int u = VALUES; u < 3; ++u) ok = ok && __float_as_uint(x.v[u]) == t;
  return ok;
}

// A block's geometry and where its rows lie in shared memory.  Per field f, at
// f * kFieldFloats (a constant, so that one address register serves all fields):
// the rows of slot 0, of slot 1 (NI * NJ each), then the halo rows: the plane
// before and the plane after (NJ + 2 rows each), then rows j0-1 and j0+nj of every
// own plane.  The sponge rows (N4 floats each) follow the fields.  A row holds N
// cells with the cell after the last at [N] and the one before the first at [-1],
// so a thread's k neighbours lie beside its cells, wrap or not.
struct Block {
  int N, N4, RS, NI, NJ, NJ2, SLOT;
  int i0, j0, ni, nj;
};

// Floats of a field's rows, at most: two slots and the halo.  COMPLEX 96^3 in 12 x
// 12 blocks takes 4 + 164 rows of 100 floats = 16404; REAL 108^3 4 + 202 rows of
// 112 = 22628.  SMALL: lattices of up to 36^3 (4 + 34 rows of 40 = 1364), whose blocks of
// 192 threads or fewer leave an SM registers for another's, so that runs on several
// streams share the chip (with 180 KB a block one waited for the other's whole launch).
template <int LEVEL, bool SMALL>
constexpr int kFieldFloats = SMALL ? 1376 : LEVEL == LFM_REAL ? 22656 : 16448;

// A thread's cells: k0 .. k0+V-1 of row jr, planes [pa, pb).
struct Cells {
  int jr, kg, groups, k0;
  int pa, pb;
  bool first, last;  // the row's first / last group: its end copies are this thread's
  bool edge_row;     // row 0 or nj-1 of the block
};

// Offsets of the thread's first cell in rows jr-1, jr, jr+1 of a plane.
struct RowOff {
  int m, z, p;
};

// Walks a thread's rows plane by plane: own planes lie NJ rows apart, the halo rows
// beside them (under m at row 0, under p at row nj-1) two rows apart, and the planes
// before and after the block among the halo rows.
struct RowWalk {
  RowOff next;     // of the next own plane
  int dz, dm, dp;  // to the plane after
};

__device__ __forceinline__ RowWalk walk_from(const Block& B, const Cells& T, int cur, int ii) {
  RowWalk w;
  const int halo = 4 + T.k0 + 2 * B.SLOT, side = halo + (2 * B.NJ2 + 2 * ii) * B.RS;
  w.dz = B.NJ * B.RS;
  w.dm = T.jr > 0 ? w.dz : 2 * B.RS;
  w.dp = T.jr < B.nj - 1 ? w.dz : 2 * B.RS;
  w.next.z = 4 + T.k0 + cur * B.SLOT + (ii * B.NJ + T.jr) * B.RS;
  w.next.m = T.jr > 0 ? w.next.z - B.RS : side;
  w.next.p = T.jr < B.nj - 1 ? w.next.z + B.RS : side + B.RS;
  return w;
}

__device__ __forceinline__ RowOff halo_plane(const Block& B, const Cells& T, bool after) {
  const int m = 4 + T.k0 + 2 * B.SLOT + ((after ? B.NJ2 : 0) + T.jr) * B.RS;
  return RowOff{m, m + B.RS, m + 2 * B.RS};
}

__device__ __forceinline__ RowOff step_rows(RowWalk& w) {
  const RowOff o = w.next;
  w.next.m += w.dm;
  w.next.z += w.dz;
  w.next.p += w.dp;
  return o;
}

struct Step {
  int cur;         // shared-memory slot of the current time level
  int to_prev;     // from a cell of the current slot to the other one's
  bool damp;       // previous Psi is stored undamped
  bool store;      // the new time level goes to global memory (s_dst)
  uint32_t t;      // the new time level
  ulonglong2* out; // the block's outer rows of time t in the exchange buffer
};

// Where a time level's fields go in global memory: the field slot (the last two time
// levels) and the caller's store for that level, null = nowhere.
struct Destinations {
  float* p[2][3];
};

// The place of outer row (ii, jr) of an ni x nj block among its exchanged rows.
__device__ __forceinline__ int outer_row(int ii, int jr, int ni, int nj, int NI, int NJ) {
  if (ii == 0) return jr;
  if (ii == ni - 1) return NJ + jr;
  return 2 * NJ + (jr == 0 ? 0 : NI) + ii;
}

template <int V>
__device__ __forceinline__ void load_rows(QPlane<V>& q, const float* f, const RowOff& o) {
  q.m = lds<V>(f, o.m);
  q.z = lds<V>(f, o.z);
  q.p = lds<V>(f, o.p);
  q.zl = f[o.z - 1];
  q.zr = f[o.z + V];
}

template <int V>
__device__ __forceinline__ void load_sides(QPlane<V>& q, const float* f, const RowOff& o) {
  q.ml = f[o.m - 1];
  q.mr = f[o.m + V];
  q.pl = f[o.p - 1];
  q.pr = f[o.p + V];
}

// Stores a thread's two values at its place `p` of a row in global memory.  EVEN: N
// is even, so the row's last group has both cells and rows start on 8 bytes.
template <bool EVEN>
__device__ __forceinline__ void store_global(float* p, const float (&x)[2], const Cells& T) {
  if constexpr (EVEN) {
    stg<2>(p, x);
  } else {
    p[0] = x[0];
    if (!T.last) p[1] = x[1];
  }
}

// The same in shared memory, with the copies beyond the row's ends.
template <bool EVEN>
__device__ __forceinline__ void store_row(float* p, const float (&x)[2], const Block& B,
                                          const Cells& T) {
  if (EVEN || !T.last)
    stg<2>(p, x);
  else
    p[0] = x[0];
  if (T.first) p[B.N] = x[0];
  if (T.last) p[-T.k0 - 1] = EVEN ? x[1] : x[0];
}

template <int LEVEL, bool EVEN, bool SMALL, int PA, int PB, int PC>
__device__ __forceinline__ void plane(const StepConsts& c, float* sm, const Block& B,
                                      const Cells& T, const Step& S,
                                      QPlane<kCells> (&Q)[kFields<LEVEL>][3], int ii,
                                      RowOff& centre, RowWalk& walk, int& mask_at,
                                      const Destinations& D) {
  constexpr int NS = kFields<LEVEL>, FS = kFieldFloats<LEVEL, SMALL>, V = kCells;
  const RowOff nxt = ii + 1 < B.ni ? walk.next : halo_plane(B, T, true);
  step_rows(walk);
#pragma unroll
  for (int f = 0; f < NS; ++f) {
    load_rows<V>(Q[f][PC], sm + f * FS, nxt);
    load_sides<V>(Q[f][PB], sm + f * FS, centre);
  }
  const int prv = centre.z + S.to_prev;
  const Vec<V> mask = lds<V>(sm + NS * FS, mask_at);
  mask_at += B.NJ * B.N4;
  Vec<V> old[NS];
#pragma unroll
  for (int f = 0; f < NS; ++f) old[f] = lds<V>(sm + f * FS, prv);
  float out[NS][V];
#pragma unroll
  for (int e = 0; e < V; e += 2) {
    const F2 mk = pk(mask.v[e], mask.v[e + 1]);
    const F2 ab = fsub(cst<F2>(1.0f), mk);
    const S19 X0 = q_s19<V>(Q[NS - 1][PA], Q[NS - 1][PB], Q[NS - 1][PC], e);
    const S19 X1 = q_s19<V>(Q[NS - 1][PA], Q[NS - 1][PB], Q[NS - 1][PC], e + 1);
    const F2 xp = pk(old[NS - 1].v[e], old[NS - 1].v[e + 1]);
    const S19 R0 = q_s19<V>(Q[0][PA], Q[0][PB], Q[0][PC], e);
    const S19 R1 = q_s19<V>(Q[0][PA], Q[0][PB], Q[0][PC], e + 1);
    F2 rp = pk(old[0].v[e], old[0].v[e + 1]);
    if (S.damp) rp = fmul(rp, ab);
    if constexpr (LEVEL == LFM_REAL) {
      const RealOutT<F2> o = real_cell_ab(lap19_pair(R0, R1), pk(R0.c, R1.c), rp,
                                          lap19_pair(X0, X1), pk(X0.c, X1.c), xp, mk, ab, c);
      out[0][e] = o.psi.v.x; out[0][e + 1] = o.psi.v.y;
      out[1][e] = o.chi.v.x; out[1][e + 1] = o.chi.v.y;
    } else {
      const S19 I0 = q_s19<V>(Q[1][PA], Q[1][PB], Q[1][PC], e);
      const S19 I1 = q_s19<V>(Q[1][PA], Q[1][PB], Q[1][PC], e + 1);
      F2 ip = pk(old[1].v[e], old[1].v[e + 1]);
      if (S.damp) ip = fmul(ip, ab);
      const ComplexOutT<F2> o = complex_cell_ab(
          lap19_pair(R0, R1), pk(R0.c, R1.c), rp, pk_faces(faces_of(R0), faces_of(R1)),
          lap19_pair(I0, I1), pk(I0.c, I1.c), ip, pk_faces(faces_of(I0), faces_of(I1)),
          lap19_pair(X0, X1), pk(X0.c, X1.c), xp, mk, ab, c);
      out[0][e] = o.pr.v.x; out[0][e + 1] = o.pr.v.y;
      out[1][e] = o.pi.v.x; out[1][e + 1] = o.pi.v.y;
      out[2][e] = o.chi.v.x; out[2][e + 1] = o.chi.v.y;
    }
  }
#pragma unroll
  for (int f = 0; f < NS; ++f) store_row<EVEN>(sm + f * FS + prv, out[f], B, T);
  if (T.edge_row || ii == 0 || ii == B.ni - 1) {
    constexpr int NP = kPackets<LEVEL, V>;
    ulonglong2* d = S.out + outer_row(ii, T.jr, B.ni, B.nj, B.NI, B.NJ) * NP * T.groups + T.kg;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      Packet x;
#pragma unroll
      for (int u = 0; u < 3; ++u) {  // value 3p + u, field-major; a spare place: the time level
        const int w = 3 * p + u;
        x.v[u] = w < NS * V ? out[w / V][w % V] : __uint_as_float(S.t);
      }
      x.t = S.t;
      st_packet(d + p * T.groups, x);
    }
  }
  if (S.store) {
    const int g = ((B.i0 + ii) * B.N + B.j0 + T.jr) * B.N + T.k0;
#pragma unroll
    for (int f = 0; f < NS; ++f) {
      if (D.p[0][f]) store_global<EVEN>(D.p[0][f] + g, out[f], T);
      if (D.p[1][f]) store_global<EVEN>(D.p[1][f] + g, out[f], T);
    }
  }
  centre = nxt;
}

// Reads the halo rows of time t from the neighbours' packets into shared memory.
// A thread takes the V cells of group kg of every rows_a_round-th row, the first
// kBatch rows at once: their packets are polled before the CTA's barrier, behind
// which every thread is done with the halo of the time before.
template <int LEVEL, bool EVEN, bool SMALL>
__device__ __forceinline__ bool receive(float* sm, const Block& B, const Cells& T,
                                        const ulonglong2* in, const int* halo_src, int HR,
                                        uint32_t t, int first, int rows_a_round) {
  constexpr int V = kCells, NS = kFields<LEVEL>, NP = kPackets<LEVEL, V>, kBatch = 4;
  constexpr int FS = kFieldFloats<LEVEL, SMALL>;
  constexpr int LAST = NS * V - 3 * (NP - 1);  // values in a group's last packet
  bool ok = true, met = false;
  for (int q = first; q < HR || !met; q += kBatch * rows_a_round) {
    Packet x[kBatch][NP];
    const ulonglong2* src[kBatch];
    bool want[kBatch][NP];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int r = q + u * rows_a_round;
      const int place = r < HR ? halo_src[r] : -1;
      src[u] = in + place + T.kg;
#pragma unroll
      for (int p = 0; p < NP; ++p) want[u][p] = place >= 0;
    }
    // Every round loads all packets still missing, so that a wait costs the last
    // one's latency and not each one's.  The clock is read every 64 rounds only.
    uint64_t t0 = 0;
    for (uint32_t n = 1;; ++n) {
#pragma unroll
      for (int u = 0; u < kBatch; ++u)
#pragma unroll
        for (int p = 0; p < NP; ++p)
          if (want[u][p]) x[u][p] = ld_packet(src[u] + p * T.groups);
      bool missing = false;
#pragma unroll
      for (int u = 0; u < kBatch; ++u)
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          want[u][p] = want[u][p] && !(p < NP - 1 ? carries<3>(x[u][p], t)
                                                  : carries<LAST>(x[u][p], t));
          missing = missing || want[u][p];
        }
      if (!missing) break;
      if ((n & 63u) == 0) {
        const uint64_t now = now_ns();
        if (t0 == 0) t0 = now;
        ok = now - t0 <= kWaitLimitNs;
        if (!ok) break;
      }
    }
    if (!met) __syncthreads();
    met = true;
    if (!ok) return false;
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      if (q + u * rows_a_round >= HR || halo_src[q + u * rows_a_round] < 0) continue;
      float* row = sm + 4 + T.k0 + 2 * B.SLOT + (q + u * rows_a_round) * B.RS;
#pragma unroll
      for (int f = 0; f < NS; ++f) {
        float v[V];
#pragma unroll
        for (int e = 0; e < V; ++e) v[e] = x[u][(f * V + e) / 3].v[(f * V + e) % 3];
        store_row<EVEN>(row + f * FS, v, B, T);
      }
    }
  }
  return true;
}

template <int BYTES>
__device__ __forceinline__ void copy_async(float* dst, const float* src) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// Starts the copies of rows listed in `rows` (global row numbers, -1 = none) of one
// array into shared memory, row r at dst + 4 + r * RS; a warp takes a row.  All of a
// block's copies are in flight at once (a row's loads at a time, then its stores,
// filled a block of COMPLEX 96^3 in 50 us).
__device__ __forceinline__ void copy_rows(const float* src, float* dst, const int* rows,
                                          int count, const Block& B, int warp, int nwarps,
                                          int lane) {
  for (int r = warp; r < count; r += nwarps) {
    if (rows[r] < 0) continue;
    const float* s = src + rows[r] * B.N;
    float* d = dst + 4 + r * B.RS;
    if ((B.N & 3) == 0) {  // at most 32 groups of four
      if (4 * lane < B.N) copy_async<16>(d + 4 * lane, s + 4 * lane);
    } else {
      for (int k = lane; k < B.N; k += 32) copy_async<4>(d + k, s + k);
    }
  }
}

// The copies beyond the ends of rows [0, count) at dst, once the rows are there.
__device__ __forceinline__ void copy_ends(float* dst, int count, const Block& B) {
  for (int r = threadIdx.x; r < count; r += blockDim.x) {
    float* d = dst + 4 + r * B.RS;
    const float first = d[0], last = d[B.N - 1];
    d[B.N] = first;
    d[-1] = last;
  }
}

// The lattices of a launch: CTAs [first[l], first[l + 1]) run lattice l.
template <int LATTICES>
struct Wave {
  int count;
  int first[LATTICES + 1];
  ResidentArgs lattice[LATTICES];
};

template <int LEVEL, bool EVEN, int THREADS, int LATTICES, bool SMALL>
__global__ void __launch_bounds__(THREADS, 1)
    resident_kernel(const __grid_constant__ Wave<LATTICES> W) {
  constexpr int V = kCells, NS = kFields<LEVEL>;
  int l = 0;
  if constexpr (LATTICES > 1)
    while ((int)blockIdx.x >= W.first[l + 1]) ++l;
  const ResidentArgs& A = W.lattice[l];
  extern __shared__ __align__(16) float sm[];
  __shared__ int s_abort;
  __shared__ Destinations s_dst;
  const ResidentPlan& L = A.plan;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int b = blockIdx.x - (LATTICES > 1 ? W.first[l] : 0), bi = b / L.nbj, bj = b % L.nbj;
  Block B;
  B.N = A.N;
  B.N4 = (A.N + 3) & ~3;
  B.RS = L.RS;
  B.NI = L.NI;
  B.NJ = L.NJ;
  B.NJ2 = L.NJ + 2;
  B.SLOT = L.NI * L.NJ * L.RS;
  const int HR = 2 * B.NJ2 + 2 * L.NI;  // halo rows of a field
  B.i0 = bi * A.N / L.nbi;
  B.ni = (bi + 1) * A.N / L.nbi - B.i0;
  B.j0 = bj * A.N / L.nbj;
  B.nj = (bj + 1) * A.N / L.nbj - B.j0;
  constexpr int FS = kFieldFloats<LEVEL, SMALL>;
  float* mask_rows = sm + NS * FS;
  int* halo_row = reinterpret_cast<int*>(mask_rows + L.NI * L.NJ * B.N4);  // HR entries
  int* own_row = halo_row + HR;                                // NI * NJ entries
  int* halo_src = own_row + L.NI * L.NJ;  // HR entries: the row's packets in a buffer
  constexpr int NP = kPackets<LEVEL, V>;
  const int groups = (A.N + V - 1) / V;
  const int OR = 2 * L.NI + 2 * L.NJ;  // exchanged rows of a block

  // ---- load -----------------------------------------------------------------
  auto wrap = [&](int x) { return x < 0 ? x + A.N : (x >= A.N ? x - A.N : x); };
  for (int q = tid; q < HR; q += blockDim.x) {
    int ii, jj;
    bool used;
    if (q < 2 * B.NJ2) {
      const int s = q / B.NJ2;
      ii = s ? B.ni : -1;
      jj = q - s * B.NJ2 - 1;
      used = jj <= B.nj;
    } else {
      ii = (q - 2 * B.NJ2) >> 1;
      jj = (q & 1) ? B.nj : -1;
      used = ii < B.ni;
    }
    halo_row[q] = used ? wrap(B.i0 + ii) * A.N + wrap(B.j0 + jj) : -1;
    int src = -1;
    if (used) {  // the owner's block and the row's place in it
      int oi = bi + (ii < 0 ? -1 : (ii == B.ni ? 1 : 0)), oj = bj + (jj < 0 ? -1 : (jj == B.nj ? 1 : 0));
      oi = oi < 0 ? L.nbi - 1 : (oi == L.nbi ? 0 : oi);
      oj = oj < 0 ? L.nbj - 1 : (oj == L.nbj ? 0 : oj);
      const int a0 = oi * A.N / L.nbi, an = (oi + 1) * A.N / L.nbi - a0;
      const int b0 = oj * A.N / L.nbj, bn = (oj + 1) * A.N / L.nbj - b0;
      const int row = outer_row(wrap(B.i0 + ii) - a0, wrap(B.j0 + jj) - b0, an, bn, L.NI, L.NJ);
      src = ((oi * L.nbj + oj) * OR + row) * NP * groups;
    }
    halo_src[q] = src;
  }
  for (int r = tid; r < L.NI * L.NJ; r += blockDim.x) {
    const int ii = r / L.NJ, jj = r % L.NJ;
    own_row[r] = ii < B.ni && jj < B.nj ? (B.i0 + ii) * A.N + B.j0 + jj : -1;
  }
  if (tid == 0) s_abort = 0;
  const uint32_t base = *reinterpret_cast<volatile uint32_t*>(A.sync);
  __syncthreads();
#pragma unroll
  for (int f = 0; f < NS; ++f) {
    float* d = sm + f * FS;
    copy_rows(A.cur[f], d, own_row, L.NI * L.NJ, B, warp, nwarps, lane);
    copy_rows(A.prev[f], d + B.SLOT, own_row, L.NI * L.NJ, B, warp, nwarps, lane);
    copy_rows(A.cur[f], d + 2 * B.SLOT, halo_row, HR, B, warp, nwarps, lane);
  }
  for (int r = warp; r < L.NI * L.NJ; r += nwarps) {
    const int q = qterm(B.i0 + r / L.NJ, A.N) + qterm(B.j0 + r % L.NJ, A.N);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = lane + 32 * u;
      if (k < B.N4)
        mask_rows[r * B.N4 + k] = mask_from_q_flat(A.lut, q + qterm(k < A.N ? k : 0, A.N));
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int f = 0; f < NS; ++f) copy_ends(sm + f * FS, 2 * L.NI * L.NJ + HR, B);

  Cells T;
  T.groups = groups;
  T.kg = tid % groups;
  const int per_seg = B.nj * groups;
  const int seg = tid / per_seg;
  const bool active = seg < L.segs;
  T.jr = (tid - seg * per_seg) / groups;
  T.k0 = T.kg * V;  // per_seg is a multiple of groups
  T.first = T.kg == 0;
  T.last = T.kg == groups - 1;
  T.edge_row = T.jr == 0 || T.jr == B.nj - 1;
  T.pa = active ? seg * B.ni / L.segs : 0;
  T.pb = active ? (seg + 1) * B.ni / L.segs : 0;
  const int rows_a_round = blockDim.x / groups;
  const int first_row = tid / groups < rows_a_round ? tid / groups : HR;
  const int64_t buffer = (int64_t)L.nbi * L.nbj * OR * NP * groups;  // packets of a time level
  // one thread a destination of the time level that step s makes
  const auto set_destination = [&](int s) {
    if (tid >= 2 * NS) return;
    const int f = tid % NS;
    float* p = nullptr;
    if (tid < NS)
      p = s >= A.steps - 2 ? ((s & 1) ? A.even[f] : A.odd[f]) : nullptr;
    else if (A.stores)
      p = A.stores[s * NS + f];
    s_dst.p[tid / NS][f] = p;
  };
  // whether step s may store: the destinations are looked at only then (the reads
  // cost REAL 32^3 7 % of its step)
  const auto stores = [&](int s) { return A.stores != nullptr || s >= A.steps - 2; };
  set_destination(0);
  __syncthreads();

  // ---- steps ----------------------------------------------------------------
  for (int s = 0; s < A.steps; ++s) {
    Step S;
    S.cur = s & 1;
    S.to_prev = (1 - 2 * S.cur) * B.SLOT;
    S.damp = s > 0 || A.damp_first;
    S.store = stores(s);
    S.t = base + (uint32_t)(s + 1);
    ulonglong2* packets = A.packets + (S.t & 1u) * buffer;
    S.out = packets + (int64_t)b * OR * NP * groups;
    if (T.pa < T.pb) {
      QPlane<V> Q[NS][3];
      RowWalk walk = walk_from(B, T, S.cur, T.pa > 0 ? T.pa - 1 : 0);
      RowOff centre = T.pa > 0 ? step_rows(walk) : halo_plane(B, T, false);
#pragma unroll
      for (int f = 0; f < NS; ++f) load_rows<V>(Q[f][0], sm + f * FS, centre);
      centre = step_rows(walk);
#pragma unroll
      for (int f = 0; f < NS; ++f) load_rows<V>(Q[f][1], sm + f * FS, centre);
      int ii = T.pa, mask_at = (T.pa * B.NJ + T.jr) * B.N4 + T.k0;
      while (true) {
        plane<LEVEL, EVEN, SMALL, 0, 1, 2>(A.c, sm, B, T, S, Q, ii, centre, walk, mask_at, s_dst);
        if (++ii >= T.pb) break;
        plane<LEVEL, EVEN, SMALL, 1, 2, 0>(A.c, sm, B, T, S, Q, ii, centre, walk, mask_at, s_dst);
        if (++ii >= T.pb) break;
        plane<LEVEL, EVEN, SMALL, 2, 0, 1>(A.c, sm, B, T, S, Q, ii, centre, walk, mask_at, s_dst);
        if (++ii >= T.pb) break;
      }
    }
    if (s + 1 == A.steps) break;
    if (!receive<LEVEL, EVEN, SMALL>(sm, B, T, packets, halo_src, HR, S.t, first_row,
                                     rows_a_round)) {
      s_abort = 1;
      atomicOr(A.status, LFM_ERR_DEVICE_TIMEOUT);
    }
    if (stores(s + 1)) set_destination(s + 1);  // behind receive()'s barrier: step s has stored
    __syncthreads();
    if (s_abort) break;
  }
  // The last CTA to retire moves the time base on for the next launch.
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(A.sync + 1, 1u) == gridDim.x - 1) {
      atomicExch(A.sync + 1, 0u);
      atomicExch(A.sync, base + (uint32_t)A.steps);
    }
  }
}

template <int LEVEL, bool EVEN, int THREADS, int LATTICES, bool SMALL>
cudaError_t launch(const Wave<LATTICES>& w, int threads, int smem, cudaStream_t stream) {
  static SmemGrant grant;
  const auto kernel = resident_kernel<LEVEL, EVEN, THREADS, LATTICES, SMALL>;
  const cudaError_t e = grant.raise((const void*)kernel, smem);
  if (e != cudaSuccess) return e;
  void* args[] = {const_cast<Wave<LATTICES>*>(&w)};
  return cudaLaunchCooperativeKernel((const void*)kernel, dim3(w.first[w.count]), dim3(threads),
                                     args, (size_t)smem, stream);
}

template <int LEVEL, bool EVEN>
cudaError_t launch_level(const ResidentArgs& a, cudaStream_t stream) {
  Wave<1> w{1, {0, a.plan.nbi * a.plan.nbj}, {a}};
  const int t = a.plan.threads, sm = a.plan.smem;
  static_assert(kThreadsComplex == 384, "one block size for COMPLEX and the smaller REAL blocks");
  if (a.plan.small) return launch<LEVEL, EVEN, 384, 1, true>(w, t, sm, stream);
  if constexpr (LEVEL == LFM_REAL)
    if (t > 384) return launch<LEVEL, EVEN, 512, 1, false>(w, t, sm, stream);
  return launch<LEVEL, EVEN, 384, 1, false>(w, t, sm, stream);
}

// Bytes of dynamic shared memory of a block: the fields, the sponge rows, the row tables.
int smem_bytes(int level, int N, int NI, int NJ, bool small) {
  const bool cx = level == LFM_COMPLEX;
  const int field = small ? kFieldFloats<LFM_REAL, true>
                          : cx ? kFieldFloats<LFM_COMPLEX, false> : kFieldFloats<LFM_REAL, false>;
  const int N4 = (N + 3) / 4 * 4, halo = 2 * (NJ + 2) + 2 * NI;
  return 4 * ((cx ? 3 : 2) * field + NI * NJ * N4 + 2 * halo + NI * NJ);
}

template <int LEVEL>
cudaError_t launch_wave(const ResidentArgs* a, int count, cudaStream_t stream) {
  static_assert(sizeof(Wave<kWaveLattices>) < 32000, "kernel parameters");
  Wave<kWaveLattices> w{};
  w.count = count;
  int threads = 0, smem = 0;
  for (int l = 0; l < count; ++l) {
    w.lattice[l] = a[l];
    w.first[l + 1] = w.first[l] + a[l].plan.nbi * a[l].plan.nbj;
    threads = std::max(threads, a[l].plan.threads);
    smem = std::max(smem, smem_bytes(LEVEL, a[l].N, a[l].plan.NI, a[l].plan.NJ, false));
  }
  if constexpr (LEVEL == LFM_COMPLEX)
    return launch<LEVEL, true, kThreadsComplex, kWaveLattices, false>(w, threads, smem, stream);
  else
    return threads <= 384
               ? launch<LEVEL, true, 384, kWaveLattices, false>(w, threads, smem, stream)
               : launch<LEVEL, true, 512, kWaveLattices, false>(w, threads, smem, stream);
}

}  // namespace

// The cheapest cut by a model of a step in SM cycles: the march (planes of a
// segment and half a plane of start-up, each the issue of the scheduler's warps or
// one warp's own latency), the halo packets a CTA reads, and the latency of the
// exchange.  Measured on B200: a warp's plane 330 (REAL) / 480 (COMPLEX) cycles
// with several warps on the scheduler, 900 / 1200 alone; 0.7 cycles a packet; 2300
// for the exchange itself.
// When the model was fitted, the best of the cuts tried and this model's: REAL 32^3
// 2.16 / 2.23 us a step, 64^3 3.53 / 3.53, 96^3 7.5 / 7.5; COMPLEX 64^3 4.37 / 4.40,
// 96^3 9.2 / 9.2.  The model's cuts now take 1.87, 3.23, 6.57; 3.87, 8.26 us, the
// tile kernel launched once a step 7.2, 8.7, 13.3; 9.3, 20.7.
//
// plans[c]: the cheapest cut of at most c blocks (c = 0: none), for c up to 148.
static const std::vector<ResidentPlan>& resident_plans(int level, int N) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, std::vector<ResidentPlan>> tables;  // at most 2 x 121
  std::lock_guard<std::mutex> lk(mu);
  std::vector<ResidentPlan>& plans = tables[{level, N}];
  if (!plans.empty()) return plans;
  plans.resize(kMaxBlocks + 1);
  const bool cx = level == LFM_COMPLEX;
  const int ns = cx ? 3 : 2, V = kCells, np = (ns * V + 2) / 3;
  const int RS = (N + 3) / 4 * 4 + 4;
  const int field = cx ? kFieldFloats<LFM_COMPLEX, false> : kFieldFloats<LFM_REAL, false>;
  const int groups = (N + V - 1) / V;
  for (int nbi = 1; nbi <= std::min(N, kMaxBlocks); ++nbi) {
    for (int nbj = 1; nbj <= std::min(N, kMaxBlocks / nbi); ++nbj) {
      const int NI = (N + nbi - 1) / nbi, NJ = (N + nbj - 1) / nbj;
      const int lanes = NJ * groups;
      if (lanes > kMaxThreads) continue;
      const int halo = 2 * (NJ + 2) + 2 * NI;
      const int rows = 4 + (2 * NI * NJ + halo) * RS;
      if (rows > field || smem_bytes(level, N, NI, NJ, false) > kSmemBytes) continue;
      for (int segs = 1; segs <= std::min(NI, kMaxThreads / lanes); ++segs) {
        const int warps = (segs * lanes + 31) / 32, planes = (NI + segs - 1) / segs;
        if (32 * warps > (cx ? kThreadsComplex : kMaxThreads)) break;
        const double issue = cx ? 480.0 : 330.0;
        const double t = (planes + 0.5) * std::max((warps + 3) / 4 * issue, cx ? 1200.0 : 900.0) +
                         0.7 * halo * groups * np + 2300.0;
        const bool small =
            N <= kSmallEdge && rows <= kFieldFloats<LFM_REAL, true> && 32 * warps <= 384;
        const int smem = smem_bytes(level, N, NI, NJ, small);
        ResidentPlan& best = plans[nbi * nbj];
        if (best.nbi == 0 || t < best.cycles)
          best = ResidentPlan{nbi, nbj, NI, NJ, V, segs, warps * 32, RS, smem, small,
                              4 + 8LL * nbi * nbj * 2 * (NI + NJ) * np * groups, t};
      }
    }
  }
  for (int c = 1; c <= kMaxBlocks; ++c)
    if (plans[c].nbi == 0 || (plans[c - 1].nbi && plans[c - 1].cycles <= plans[c].cycles))
      plans[c] = plans[c - 1];
  return plans;
}

bool resident_plan(int level, int N, int sms, ResidentPlan* out) {
  if ((level != LFM_REAL && level != LFM_COMPLEX) || N < 8 || N > 128 || sms < 1) return false;
  *out = resident_plans(level, N)[std::min(sms, kMaxBlocks)];
  return out->nbi > 0;
}

// Packs the lattices of one level into waves: with a step time T in mind each takes
// the fewest blocks that make a step in T (or as fast as it can), the largest go
// first into the first wave with room, and what a wave has left speeds its slowest
// lattice up.  The T of the smallest total is taken.
static void pack_level(const int* N, const std::vector<int>& idx, int level, int sms,
                         std::vector<ResidentWavePlan>* out) {
  double best_total = 1e300;
  std::vector<ResidentWavePlan> best;
  for (double T = 4000.0; T < 60000.0; T *= 1.12) {
    std::vector<std::pair<int, int>> need;  // blocks, lattice
    for (int l : idx) {
      const std::vector<ResidentPlan>& p = resident_plans(level, N[l]);
      int c = sms;
      while (c > 1 && p[c - 1].nbi && p[c - 1].cycles <= std::max(T, p[sms].cycles)) --c;
      need.push_back({p[c].nbi * p[c].nbj, l});
    }
    std::stable_sort(need.begin(), need.end(),
                     [](const auto& a, const auto& b) { return a.first > b.first; });
    std::vector<ResidentWavePlan> waves;
    for (const auto& n : need) {
      const int c = n.first, l = n.second;
      auto w = std::find_if(waves.begin(), waves.end(), [&](const ResidentWavePlan& v) {
        return v.blocks + c <= sms && (int)v.lattices.size() < kWaveLattices;
      });
      if (w == waves.end()) w = waves.insert(waves.end(), ResidentWavePlan{level, 0, {}, {}});
      w->blocks += c;
      w->lattices.push_back(l);
      w->plans.push_back(resident_plans(level, N[l])[c]);
    }
    double total = 0.0;
    for (ResidentWavePlan& w : waves) {
      while (true) {
        size_t slow = 0;
        for (size_t k = 1; k < w.plans.size(); ++k)
          if (w.plans[k].cycles > w.plans[slow].cycles) slow = k;
        const ResidentPlan& now = w.plans[slow];
        const int used = now.nbi * now.nbj;
        const ResidentPlan& more =
            resident_plans(level, N[w.lattices[slow]])[used + sms - w.blocks];
        if (more.cycles >= now.cycles) {
          total += now.cycles;
          break;
        }
        w.blocks += more.nbi * more.nbj - used;
        w.plans[slow] = more;
      }
    }
    if (total < best_total) {
      best_total = total;
      best.swap(waves);
    }
  }
  out->insert(out->end(), best.begin(), best.end());
}

bool resident_waves(const int* level, const int* N, int count, int sms,
                    std::vector<ResidentWavePlan>* waves) {
  sms = std::min(sms, kMaxBlocks);
  waves->clear();
  for (int lv : {LFM_REAL, LFM_COMPLEX}) {
    std::vector<int> idx;
    for (int l = 0; l < count; ++l) {
      ResidentPlan p;
      if (!resident_plan(level[l], N[l], sms, &p) || N[l] % 2) return false;
      if (level[l] == lv) idx.push_back(l);
    }
    if (!idx.empty()) pack_level(N, idx, lv, sms, waves);
  }
  // the most blocks first, so that a launch the device has no room for is the first one
  std::stable_sort(waves->begin(), waves->end(),
                   [](const ResidentWavePlan& a, const ResidentWavePlan& b) {
                     return a.blocks > b.blocks;
                   });
  return true;
}

cudaError_t launch_resident_wave(const ResidentArgs* a, int count, cudaStream_t stream) {
  return a[0].level == LFM_REAL ? launch_wave<LFM_REAL>(a, count, stream)
                                : launch_wave<LFM_COMPLEX>(a, count, stream);
}

cudaError_t launch_resident(const ResidentArgs& a, cudaStream_t stream) {
  const bool even = a.N % 2 == 0;
  if (a.level == LFM_REAL)
    return even ? launch_level<LFM_REAL, true>(a, stream) : launch_level<LFM_REAL, false>(a, stream);
  return even ? launch_level<LFM_COMPLEX, true>(a, stream)
              : launch_level<LFM_COMPLEX, false>(a, stream);
}

}  // namespace lfm
