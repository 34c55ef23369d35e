// Per-planet FP64 global budgets and the device-side monthly-mean
// accumulation of the published snapshot (the reference's page-side
// averager and energy balance, src/model/climate/gcm/averages/index.ts:26-142
// and balance/index.ts, moved next to the state).
//
// On every step a slot publishes, one 256-thread block per slot sums, with a
// fixed order in double precision, the Gaussian-weighted global means of
//   0 surface pressure (the atmosphere's mass, Pa)
//   1 top-of-atmosphere net radiation (W/m^2; snapshot field 16)
//   2 surface net heat flux (W/m^2; snapshot field 17)
//   3 surface temperature (K; snapshot field 0)
//   4 precipitation, convective + large-scale (m/s; snapshot field 5)
//   5 evaporation (m/s, positive upward; snapshot field 18)
//   6 column water vapour (kg/m^2; snapshot field 7)
//   7 the weights' own mean (1 up to rounding: a check)
// and keeps the last values, their running sums and the number of samples.
// The global mean is sum_h w(lat h) f(h) / sum_h w(lat h), the weights the
// FP64 Gaussian weights (summing to 2 per longitude). With averages enabled
// the same step adds every snapshot field of the slot to an FP64 running sum
// (averages/index.ts `add`); exogcm_averages_read returns sum / samples (its
// `close`).
#include <cuda_runtime.h>

#include "common.cuh"
#include "launch.h"

namespace exogcm {

namespace {

constexpr int kThreads = 256;

// A block's threads are two groups of kThreads, each summing four of the
// quantities over the points in the order one thread per point stride takes
// them (a fixed order, whatever the split), eight points in flight. With all
// eight in one group and one point at a time the block spent 55 us at T42
// waiting for 32 rounds of 12 loads.
constexpr int kGroups = 2, kPerGroup = kBudgetQuantities / kGroups, kAhead = 8;

__global__ void __launch_bounds__(kGroups* kThreads) k_budget(Model m) {
  pdl_wait();
  pdl_release();
  const Dims& d = m.d;
  const int slot = blockIdx.x;
  const StepParams& P = m.params[slot];
  if (!P.active || P.snap[2] == 0.f) return;
  const FieldPtrs& F = m.f;
  const size_t SN = (size_t)d.S * d.NHOR, base = (size_t)slot * d.NHOR;
  const int NL = d.L;
  const int group = threadIdx.x / kThreads, t = threadIdx.x % kThreads;
  double acc[kPerGroup] = {};
  for (int h0 = t; h0 < d.NHOR; h0 += kAhead * kThreads) {  // NHOR is a multiple of kAhead * kThreads
    float v[kAhead][8];
    double w[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const int h = h0 + k * kThreads;
      const size_t c = base + h;
      w[k] = m.sh.wlat[h / d.NLON];
      if (group == 0) {
        v[k][0] = F.dp[c];
        v[k][1] = F.dswfl[c];
        v[k][2] = F.dlwfl[c];
        v[k][3] = F.dsmelt[c];
        v[k][4] = F.dswfl[NL * SN + c];
        v[k][5] = F.dlwfl[NL * SN + c];
        v[k][6] = F.dshfl[c];
        v[k][7] = F.dlhfl[c];
      } else {
        v[k][0] = F.dprc[c];
        v[k][1] = F.dprl[c];
        v[k][2] = F.devap[c];
        v[k][3] = F.dqvi[c];
        v[k][4] = F.dt[NL * SN + c];
      }
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      double q[kPerGroup];
      if (group == 0) {
        q[0] = (double)v[k][0];
        q[1] = (double)v[k][1] + (double)v[k][2];
        q[2] = (double)v[k][3] * -333700000.0 + (double)v[k][4] + (double)v[k][5] + (double)v[k][6] + (double)v[k][7];
        q[3] = 1.0;
      } else {
        q[0] = (double)v[k][4];
        q[1] = (double)v[k][0] + (double)v[k][1];
        q[2] = -(double)v[k][2];
        q[3] = (double)v[k][3];
      }
#pragma unroll
      for (int i = 0; i < kPerGroup; ++i) acc[i] += w[k] * q[i];
    }
  }
  __shared__ double red[kBudgetQuantities][kThreads];
#pragma unroll
  for (int i = 0; i < kPerGroup; ++i) red[group * kPerGroup + i][t] = acc[i];
  __syncthreads();
  for (int stride = kThreads / 2; stride > 0; stride /= 2) {
    if (t < stride)
#pragma unroll
      for (int i = 0; i < kPerGroup; ++i)
        red[group * kPerGroup + i][t] += red[group * kPerGroup + i][t + stride];
    __syncthreads();
  }
  if (threadIdx.x < kBudgetQuantities) {
    // quantity k's place in the groups: pressure, TOA, surface, weight | temperature, rain, evaporation, vapour
    constexpr int place[kBudgetQuantities] = {0, 1, 2, 4, 5, 6, 7, 3};
    const int k = threadIdx.x;
    double* b = m.budget + (size_t)slot * kBudgetStride;
    const double norm = 2.0 * d.NLON;  // sum of the weights over the grid
    const double v = red[place[k]][0] / norm;
    b[k] = v;
    b[kBudgetQuantities + k] += v;
    if (k == 0) {
      b[2 * kBudgetQuantities] += 1.0;
      if (m.avg) b[2 * kBudgetQuantities + 1] += 1.0;
    }
  }
}

// The published snapshot added to the FP64 running sums: one thread per
// point of every snapshot plane of every publishing slot.
__global__ void __launch_bounds__(kThreads) k_average_add(Model m, int planes) {
  pdl_wait();
  pdl_release();
  const Dims& d = m.d;
  const size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x;
  const size_t per_plane = (size_t)d.S * d.NHOR;
  if (i >= per_plane * planes) return;
  const int slot = (int)((i % per_plane) / d.NHOR);
  const StepParams& P = m.params[slot];
  if (!P.active || P.snap[2] == 0.f) return;
  m.avg[i] += (double)m.f.snapshot[i];
}

}  // namespace

void phy_budget(const Model& m, int snapshot_planes, cudaStream_t st) {
  step_launch(m.pdl, k_budget, m.d.S, kGroups * kThreads, 0, st, m);
  if (m.avg) {
    const size_t n = (size_t)snapshot_planes * m.d.S * m.d.NHOR;
    step_launch(m.pdl, k_average_add, (unsigned)((n + kThreads - 1) / kThreads), kThreads, 0, st, m, snapshot_planes);
  }
}

}  // namespace exogcm
