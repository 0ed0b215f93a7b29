// Many steps of one lattice held on chip in one launch (resident.cu).
#pragma once

#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "lfm_math.cuh"

namespace lfm {

// How a lattice is cut over the SMs: nbi x nbj blocks of whole k rows, block
// (bi, bj) owning planes [bi N / nbi, (bi+1) N / nbi) and rows likewise; NI x
// NJ the largest block.  A CTA's threads are `segs` plane segments x the rows
// of a plane x ceil(N / V) groups of V cells.
struct ResidentPlan {
  int nbi = 0, nbj = 0, NI = 0, NJ = 0;
  int V = 0, segs = 0, threads = 0;
  int RS = 0;    // floats of a shared-memory row
  int smem = 0;  // bytes of dynamic shared memory, of a lattice run by itself
  bool small = false;  // fields laid out for small lattices then
  long long words = 0;  // 32-bit words of the workspace: 4 counters, two exchange buffers
  double cycles = 0;    // the model's time of a step
};

// The plan of an N^3 lattice at `level` on `sms` SMs; false if its state does
// not fit on chip.
bool resident_plan(int level, int N, int sms, ResidentPlan* plan);

struct ResidentArgs {
  int level, N;
  int steps, damp_first;
  ResidentPlan plan;
  // Psi_r, (Psi_i,) chi at the current time level and the one before.  The last
  // two time levels go to even / odd by their distance from the current one (the
  // two-slot layout: even = cur, odd = prev), unless null; the level that step s
  // makes also goes to stores[s * fields + f] (device memory), where stores and
  // the entry are not null.
  const float* cur[3];
  const float* prev[3];
  float* even[3];
  float* odd[3];
  float* const* stores;
  StepConsts c;
  MaskLut lut;
  uint32_t* sync;        // workspace words 0 (time base) and 1 (retired CTAs)
  ulonglong2* packets;   // the two exchange buffers, from workspace word 4 on
  int* status;
};

cudaError_t launch_resident(const ResidentArgs& a, cudaStream_t stream);

// Lattices of one level that run side by side in one launch, each on its own blocks.
struct ResidentWavePlan {
  int level, blocks;
  std::vector<int> lattices;
  std::vector<ResidentPlan> plans;
};
constexpr int kWaveLattices = 32;  // at most, in a wave

// The waves that run `count` lattices on chip one wave after another, those of the most
// blocks first; false if a lattice does not fit or its N is odd.
bool resident_waves(const int* level, const int* N, int count, int sms,
                    std::vector<ResidentWavePlan>* waves);

// One wave: the same steps, sync and status for all; packets apart.
cudaError_t launch_resident_wave(const ResidentArgs* a, int count, cudaStream_t stream);

}  // namespace lfm
