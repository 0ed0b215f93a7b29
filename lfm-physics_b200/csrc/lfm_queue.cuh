// Register queue of the marching step kernels (step_tma.cu, resident.cu): the
// vector loads, the three-plane queue of a thread's cells and the neighbourhood
// it spells out, and the clock of the bounded waits.
#pragma once

#include <cstdint>

#include "lfm_cells.cuh"

namespace lfm {

constexpr uint64_t kWaitLimitNs = 1000000000ull;  // 1 s per wait

__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// ---- vector helpers ------------------------------------------------------------
template <int V>
struct Vec {
  float v[V];
};

template <int V>
__device__ __forceinline__ Vec<V> lds(const float* smem, int off) {
  Vec<V> r;
  if constexpr (V == 4) {
    const float4 t = *reinterpret_cast<const float4*>(smem + off);
    r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
  } else if constexpr (V == 2) {
    const float2 t = *reinterpret_cast<const float2*>(smem + off);
    r.v[0] = t.x; r.v[1] = t.y;
  } else {
    r.v[0] = smem[off];
  }
  return r;
}

template <int V>
__device__ __forceinline__ void stg(float* p, const float (&x)[V]) {
  if constexpr (V == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
  } else if constexpr (V == 2) {
    *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
  } else {
    *p = x[0];
  }
}

// Rows j-1, j, j+1 of one plane at a thread's V cells, and what borders them.
template <int V>
struct QPlane {
  Vec<V> m, z, p;        // rows j-1, j, j+1
  float zl, zr;          // row j at k0-1, k0+V
  float ml, mr, pl, pr;  // rows j-1, j+1 at k0-1, k0+V (loaded when centre)
};

template <int V>
__device__ __forceinline__ S19 q_s19(const QPlane<V>& M, const QPlane<V>& A, const QPlane<V>& P,
                                     int e) {
  S19 s;
  s.c = A.z.v[e];
  s.im = M.z.v[e];
  s.ip = P.z.v[e];
  s.jm = A.m.v[e];
  s.jp = A.p.v[e];
  s.km = e > 0 ? A.z.v[e - 1] : A.zl;
  s.kp = e < V - 1 ? A.z.v[e + 1] : A.zr;
  s.imjm = M.m.v[e];
  s.imjp = M.p.v[e];
  s.ipjm = P.m.v[e];
  s.ipjp = P.p.v[e];
  s.imkm = e > 0 ? M.z.v[e - 1] : M.zl;
  s.imkp = e < V - 1 ? M.z.v[e + 1] : M.zr;
  s.ipkm = e > 0 ? P.z.v[e - 1] : P.zl;
  s.ipkp = e < V - 1 ? P.z.v[e + 1] : P.zr;
  s.jmkm = e > 0 ? A.m.v[e - 1] : A.ml;
  s.jmkp = e < V - 1 ? A.m.v[e + 1] : A.mr;
  s.jpkm = e > 0 ? A.p.v[e - 1] : A.pl;
  s.jpkp = e < V - 1 ? A.p.v[e + 1] : A.pr;
  return s;
}

__device__ __forceinline__ Faces faces_of(const S19& s) {
  Faces f;
  f.im = s.im; f.ip = s.ip; f.jm = s.jm; f.jp = s.jp; f.km = s.km; f.kp = s.kp;
  return f;
}

}  // namespace lfm
