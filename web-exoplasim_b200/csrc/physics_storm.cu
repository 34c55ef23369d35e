// hurricanestep: the storm-climatology diagnostics of one column
// (physics/storm/wgsl/storm.wgsl:1-208, after ExoPlaSim's hurricanemod.f90),
// run after carbonstep and before the frame out when a planet enables them
// (NSTORMDIAG, hurricane_namelist; physics/storm/index.ts:26-43).
//
// A group of lanes per column, in FP32. This file keeps CUDA's accurate exp,
// log, pow and IEEE division: the saturated-parcel and pressure solvers iterate
// to fixed tolerances, so a coarser step changes their iteration counts.
//
// The reference's WGSL pow(x, y) is undefined for x < 0; the genesis index
// raises 2 RH to the third power, and RH at the level nearest sigma 0.6 is
// negative when the model's humidity there is. powf follows the native
// Fortran's x**3.0 there (a negative cube), where a WGSL implementation's
// exp2(y log2 x) gives NaN.
#include "launch.h"
#include "physics_common.cuh"

namespace exogcm {
namespace {

// hurricanemod.f90's fixed thermodynamic constants (storm.wgsl:6-11).
constexpr float kCpd = 1005.7f;
constexpr float kCl = 2500.0f;
constexpr float kRvp = 461.5f;
constexpr float kAlv0 = 2.501e6f;
constexpr float kCpvmcl = -630.0f;

struct Cape {
  float energy, temperature, pressure;
};

// Saturation vapour pressure (hPa) at tc degrees Celsius.
__device__ __forceinline__ float es(float tc) { return 6.112f * expf(17.67f * tc / (243.5f + tc)); }

// Vapour pressure from mixing ratio r at pressure p.
__device__ __forceinline__ float vapor(float r, float p, float rd) { return r * p / (rd / kRvp + r); }

// Mixing ratio from vapour pressure e at pressure p.
__device__ __forceinline__ float mixing(float e, float p, float rd) { return (rd / kRvp) * e / (p - e); }

// Density temperature of temperature t, total water rt and vapour r.
__device__ __forceinline__ float density(float t, float rt, float r, float rd) {
  return t * (1.0f + r / (rd / kRvp)) / (1.0f + rt);
}

// Moist entropy of temperature t, mixing ratio r and pressure p.
__device__ __forceinline__ float entropy(float t, float r, float p, float rd) {
  const float e = vapor(r, p, rd);
  const float rh = fminf(e / es(t - 273.15f), 1.0f);
  const float lv = kAlv0 + kCpvmcl * (t - 273.15f);
  const float dry = (kCpd + r * kCl) * logf(t) - rd * logf(p - e);
  if (r == 0.0f) return dry;
  return dry + lv * r / t - r * kRvp * logf(rh);
}

// A group of lanes solves one column: the lanes of a level of a parcel. NL
// levels by two parcels (the pressure loop's environmental and saturated
// one) take a half-warp at five levels and a warp at ten.
template <int NL>
struct Group {
  static constexpr int LANES = NL <= 8 ? 16 : 32;
  static_assert(2 * NL <= LANES, "two parcels' levels fit a group");
};

// Reversible-ascent CAPE of the parcel (tp, rp, pp) through the sounding
// (storm.wgsl:56-126): levels top (0) to bottom (NL - 1). The saturated
// ascent of a level starts from the level's own temperature, so the levels
// are independent: each lane of the parcel takes one (`level`; lanes outside
// have active = false) and every lane then forms the same sums from all of
// them. `first` is the warp lane of the parcel's level 0, `mask` the group's
// lanes; st, sr, sp are the column in shared memory, `kBlockCols` apart.
constexpr int kBlockCols = 32;

template <int NL>
__device__ Cape cape(const float* st, const float* sr, const float* sp, float tp, float rp, float pp, float rd,
                     int level, bool active, int first, unsigned mask) {
  const bool parcel = !(rp < 1e-6f || tp < 200.0f || pp <= 0.0f);
  float buoyancy = 0.0f;
  int stopped = 0;  // 1: at this level's temperature; 2: at the bottom's
  if (active && parcel) {
    const float rh = fminf(vapor(rp, pp, rd) / es(tp - 273.15f), 1.0f);
    const float parcel_entropy = entropy(tp, rp, pp, rd);
    const float plcl = pp * powf(rh, tp / (1669.0f - 122.0f * rh - tp));
    const float spl = sp[level * kBlockCols], stl = st[level * kBlockCols], srl = sr[level * kBlockCols];
    float tg, rg = rp;
    if (spl >= plcl) {
      tg = tp * powf(spl / pp, rd / kCpd);
    } else {
      // Saturated ascent: Newton steps on the parcel's entropy, 0.3 of a
      // step for the first two, until the temperature moves by 0.001 K.
      float next = stl;
      tg = 0.0f;
      int count = 0;
      while (!(fabsf(next - tg) <= 0.001f)) {
        tg = next;
        const float tc = tg - 273.15f;
        const float enew = es(tc);
        rg = mixing(enew, spl, rd);
        ++count;
        const float lv = kAlv0 + kCpvmcl * tc;
        const float sl = (kCpd + rp * kCl + lv * lv * rg / (kRvp * tg * tg)) / tg;
        const float em = vapor(rg, spl, rd);
        if (spl - em <= 0.0f || tg <= 0.0f) {
          stopped = 1;
          break;
        }
        const float sg = (kCpd + rp * kCl) * logf(tg) - rd * logf(spl - em) + lv * rg / tg;
        next = tg + (count < 3 ? 0.3f : 1.0f) * (parcel_entropy - sg) / sl;
        if (count > 500 || enew > spl - 1.0f || !(next > 0.0f)) {
          stopped = 2;
          break;
        }
      }
    }
    buoyancy = density(tg, rp, rg, rd) - density(stl, srl, srl, rd);
  }
  __syncwarp(mask);
  // The routine goes up from the bottom and ends at the first level that
  // stops.
  const unsigned at_level = (__ballot_sync(mask, stopped == 1) >> first) & ((1u << NL) - 1u);
  const unsigned at_bottom = (__ballot_sync(mask, stopped == 2) >> first) & ((1u << NL) - 1u);
  const unsigned rising = (__ballot_sync(mask, buoyancy > 0.0f) >> first) & ((1u << NL) - 1u);
  // Each lane forms the area between its level and the one below; the sum
  // takes them from the bottom up.
  const int below = min(level + 1, NL - 1);
  const float below_b = __shfl_sync(mask, buoyancy, first + below);
  const float p_here = sp[level * kBlockCols], p_below = sp[below * kBlockCols];
  const float slab = rd * (buoyancy + below_b) * (p_below - p_here) / (p_here + p_below);
  const int inb = rising ? min(__ffs(rising) - 1, NL - 1) : NL - 1;
  float area = 0.0f;
#pragma unroll
  for (int l = NL - 2; l >= 0; --l) {
    const float v = __shfl_sync(mask, slab, first + l);
    if (l >= inb) area += v;
  }
  const float b_bottom = __shfl_sync(mask, buoyancy, first + NL - 1);
  const float b1 = __shfl_sync(mask, buoyancy, first + inb), b0 = __shfl_sync(mask, buoyancy, first + max(inb - 1, 0));
  if (!parcel) return {0.0f, -1.0f, -1.0f};
  if (at_level > at_bottom) return {0.0f, st[(31 - __clz(at_level)) * kBlockCols], -1.0f};
  if (at_bottom) return {0.0f, st[(NL - 1) * kBlockCols], sp[(NL - 1) * kBlockCols]};
  auto T = [&](int l) { return st[l * kBlockCols]; };
  auto Pr = [&](int l) { return sp[l * kBlockCols]; };
  if (inb == NL - 1) return {0.0f, T(NL - 1), 0.0f};
  area += rd * (pp - Pr(NL - 1)) / (pp + Pr(NL - 1)) * b_bottom;
  float tob = T(inb), lnb = Pr(inb);
  if (inb > 0) {
    lnb = (Pr(inb - 1) * b1 - Pr(inb) * b0) / (b1 - b0);
    area += rd * b1 * (Pr(inb) - lnb) / (Pr(inb) + lnb);
    tob = (T(inb) * (lnb - Pr(inb - 1)) + T(inb - 1) * (Pr(inb) - lnb)) / (Pr(inb) - Pr(inb - 1));
  }
  return {fmaxf(area, 0.0f), tob, lnb};
}

// Real part of the principal cube root in hurricanemod's ventilation-
// reduced intensity: zero at VI = 0 and for |VI| >= VITHRESH.
__device__ __forceinline__ float reduced(float vi, float vithresh) {
  if (vi == 0.0f || fabsf(vi) >= vithresh) return 0.0f;
  return 2.0f / sqrtf(3.0f) * cosf(acosf(-vi / vithresh) / 3.0f);
}

// A block takes kBlockCols columns: its first warp reads them and forms what
// takes a few operations, the groups of every warp then solve the columns
// that need it, each taking the next one as it finishes (a column's pressure
// loop takes from 2 to 201 passes of two ascents), and the first warp writes
// the results. One thread per column, its levels and parcels one after the
// other, waited for the slowest of 32 columns and for that column's chain of
// up to 201 x 2 x NL Newton solves: 448 us for 7 T42 L5 planets against 210.
template <int NL>
__global__ void __launch_bounds__(kBlock) k_storm(Model m, const PlanetConst* __restrict__ pcr,
                                                  const float* __restrict__ tabr) {
  using G = Group<NL>;
  __shared__ float s_t[NL][kBlockCols], s_r[NL][kBlockCols], s_p[NL][kBlockCols];
  __shared__ float s_sst[kBlockCols], s_msl[kBlockCols], s_vmax[kBlockCols];
  __shared__ float s_energy[kBlockCols], s_pressure[kBlockCols];
  __shared__ int s_column[kBlockCols], s_count, s_next;
  pdl_wait();
  pdl_release();
  const Dims& d = m.d;
  const int slot = blockIdx.x * kBlockCols / d.NHOR;  // kBlockCols divides NHOR
  const StepParams& P = m.params[slot];
  if (!P.active) return;
  const PlanetConst& K = pcr[slot];
  if (K.NSTORMDIAG <= 0.0f) return;
  const float* tb = tabr + (size_t)slot * m.to.stride;
  const size_t SN = (size_t)d.S * d.NHOR;
  const FieldPtrs& F = m.f;
  const float* sg = tb + m.to.sigma;
  const float rd = K.GASCON;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * kBlockCols + lane;
  constexpr int bottom = NL - 1;
  float deficit = 1.0f, shear = 0.0f, vort = 0.0f;
  int i600 = 0;
  if (warp == 0) {
    int i850 = 0, i200 = 0;
    bool cold = false;
    const float msl = F.dp[c] * 0.01f;
    const float sst = F.dt[NL * SN + c];
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      const float t = F.dt[l * SN + c];
      s_t[l][lane] = t;
      s_r[l][lane] = F.dq[l * SN + c];
      s_p[l][lane] = msl * sg[l];
      cold = cold || t <= 100.0f;
      if (fabsf(sg[l] - 0.6f) < fabsf(sg[i600] - 0.6f)) i600 = l;
      if (fabsf(sg[l] - 0.85f) < fabsf(sg[i850] - 0.85f)) i850 = l;
      if (fabsf(sg[l] - 0.2f) < fabsf(sg[i200] - 0.2f)) i200 = l;
    }
    const float u850 = F.du[i850 * SN + c], v850 = F.dv[i850 * SN + c];
    const float u200 = F.du[i200 * SN + c], v200 = F.dv[i200 * SN + c];
    const float lowwind = sqrtf(u850 * u850 + v850 * v850), highwind = sqrtf(u200 * u200 + v200 * v200);
    shear = fabsf(highwind - lowwind);
    vort = F.gz[i850 * SN + c] * K.WW;
    if (s_r[i600][lane] > 0.0f && s_r[bottom][lane] > 0.0f) {
      const float t600 = s_t[i600][lane], p600 = s_p[i600][lane];
      const float smr = mixing(es(t600 - 273.15f), p600, rd);
      const float sms = entropy(t600, smr, p600, rd);
      const float sme = entropy(t600, fminf(s_r[i600][lane], smr), p600, rd);
      const float smb = entropy(sst, F.dq[NL * SN + c], msl, rd);
      const float smo = entropy(sst, mixing(es(sst - 273.15f), msl, rd), msl, rd);
      if (smo != smb) deficit = (sms - sme) / (smo - smb);
    }
    s_sst[lane] = sst;
    s_msl[lane] = msl;
    s_vmax[lane] = s_energy[lane] = s_pressure[lane] = -1.0f;
    const bool solve = sst > 278.15f && !cold && msl > 0.0f;
    const unsigned list = __ballot_sync(0xffffffffu, solve);
    if (solve) s_column[__popc(list & ((1u << lane) - 1u))] = lane;
    if (lane == 0) {
      s_count = __popc(list);
      s_next = 0;
    }
  }
  __syncthreads();
  {
    const int start = lane / G::LANES * G::LANES, sub = lane - start;
    const unsigned mask = G::LANES == 32 ? 0xffffffffu : 0xffffu << start;
    const bool active = sub < 2 * NL;
    const int parcel = active ? sub / NL : 0, level = active ? sub % NL : 0;
    const int first = start + parcel * NL;
    for (;;) {
      int next_column = 0;
      if (sub == 0) next_column = atomicAdd(&s_next, 1);
      next_column = __shfl_sync(mask, next_column, start);
      if (next_column >= s_count) break;
      const int col = s_column[next_column];
      const float *st = &s_t[0][col], *sr = &s_r[0][col], *sp = &s_p[0][col];
      const float sst = s_sst[col], msl = s_msl[col];
      const float tbot = st[bottom * kBlockCols], rbot = sr[bottom * kBlockCols];
      const Cape environmental =
          cape<NL>(st, sr, sp, tbot, rbot, sp[bottom * kBlockCols], rd, level, active && parcel == 0, start, mask);
      float vmax = -1.0f;
      // Minimum central pressure: 970 hPa first, 1000 hPa parcel cap, until
      // it moves by 0.5 hPa; bail out after 201 passes or below 400 hPa. A
      // pressure seen before repeats the passes since, none of which ended
      // the loop, until the 201st: it bails out there and then.
      float pm = 970.0f, old = pm, next = 0.0f, capem = 0.0f, capems = 0.0f, ratio = 1.0f, seen = 0.0f;
      bool failed = false;
      int count = 0;
      while (!(fabsf(next - old) <= 0.5f)) {
        if (count > 0 && pm == seen) {
          failed = true;
          break;
        }
        if ((count & (count - 1)) == 0) seen = pm;
        const float pp = fminf(pm, 1000.0f);
        const float rp = (rd / kRvp) * rbot * msl / (pp * (rd / kRvp + rbot) - rbot * msl);
        const float rs = mixing(es(sst - 273.15f), pp, rd);
        const Cape mine = cape<NL>(st, sr, sp, parcel == 0 ? tbot : sst, parcel == 0 ? rp : rs, pp, rd, level, active,
                                   first, mask);
        capem = __shfl_sync(mask, mine.energy, start);
        capems = __shfl_sync(mask, mine.energy, start + NL);
        ratio = sst / __shfl_sync(mask, mine.temperature, start + NL);
        const float tvav = 0.5f * (density(tbot, rbot, rbot, rd) + density(sst, rs, rs, rd));
        const float cat =
            fmaxf((capem - environmental.energy) + 0.5f * K.CKCD * ratio * (capems - capem), 0.0f);
        next = msl * expf(-cat / (rd * tvav));
        old = pm;
        pm = next;
        ++count;
        if (count > 200 || pm < 400.0f || !(pm > 0.0f)) {
          failed = true;
          break;
        }
      }
      if (!failed) vmax = sqrtf(fmaxf(0.0f, K.CKCD * ratio * fmaxf(0.0f, capems - capem)));
      if (sub == 0) {
        s_vmax[col] = vmax;
        s_energy[col] = environmental.energy;
        s_pressure[col] = environmental.pressure;
      }
    }
  }
  __syncthreads();
  if (warp != 0) return;
  const float vmax = s_vmax[lane];
  const float vi = vmax > 0.0f ? shear * deficit / vmax : 1.0f;
  const float rh = vapor(s_r[i600][lane], s_p[i600][lane], rd) / es(s_t[i600][lane] - 273.15f);
  const float v70 = vmax / 70.0f, damp = 1.0f + 0.1f * shear;
  const float gpi = powf(fabsf(vort * 1e5f), 1.5f) * powf(rh * 2.0f, 3.0f) * v70 * v70 * v70 / (damp * damp);
  F.capen[c] = s_energy[lane];
  F.lnb[c] = s_pressure[lane];
  F.mpoti[c] = vmax;
  F.chim[c] = deficit;
  F.laav[c] = vort;
  F.venti[c] = vi;
  F.vrmpi[c] = reduced(vi, K.VITHRESH);
  F.gpi[c] = gpi;
  F.shear[c] = shear;
}

template <int NL>
struct Storm {
  static void run(const Model& m, cudaStream_t st) {
    step_launch(m.column_pdl, k_storm<NL>, (unsigned)((size_t)m.d.S * m.d.NHOR / kBlockCols), kBlock, 0, st, m, m.pc,
                m.tabs);
  }
};

}  // namespace

void phy_storm(const Model& m, cudaStream_t st) {
  if (!m.storm) return;
  by_levels<Storm>(m.d.L, m, st);
}

}  // namespace exogcm
