// Grid-point dynamics, semi-implicit spectral update, horizontal diffusion,
// dissipative heating and the dimensional frame around the column physics,
// for every slot of a batch in one launch each (FP32).
//
// Arithmetic follows src/model/climate/gcm/dynamics/wgsl/*.wgsl (ExoPlaSim
// plasim.f90's gridpointa / spectrala / spectrald / gridpointd, in Fortran's
// statement order), with the batch's [level][slot][point] layout: column
// index c = slot * NHOR + h, spectral index c = slot * NRSP + s.
#include <cuda_runtime.h>

#include "common.cuh"
#include "launch.h"

namespace exogcm {

namespace {

constexpr int kBlock = 128;

__device__ __forceinline__ const float* slot_tabs(const Model& m, int slot) {
  return m.tabs + (size_t)slot * m.to.stride;
}

// gridpointa from gp = exp(gp) to the flux products (dynamics/wgsl/calcgp.wgsl).
// Four resident blocks per SM: a few spilled registers cost less than the
// latency the fourth block hides.
template <int NL>
__global__ void __launch_bounds__(kBlock, 4) k_calcgp(Model m) {
  pdl_wait();
  pdl_release();
  const Dims& d = m.d;
  // NHOR is a multiple of kBlock at every truncation, so a block lies in one
  // slot and that slot's vertical tables are staged in shared memory once.
  const int slot = blockIdx.x * kBlock / d.NHOR;
  if (!m.params[slot].active) return;
  __shared__ float stage[6 * NL + 2 * NL * NL];
  float* ds = stage;
  float* t0T = ds + NL;
  float* sh = t0T + NL;
  float* rd = sh + NL;
  float* t01 = rd + NL;
  float* tkpT = t01 + NL;
  float* C = tkpT + NL;
  float* G = C + NL * NL;
  {
    const float* tb = slot_tabs(m, slot);
    for (int i = threadIdx.x; i < NL * NL; i += kBlock) {
      C[i] = tb[m.to.c + i];
      G[i] = tb[m.to.g + i];
    }
    for (int i = threadIdx.x; i < NL; i += kBlock) {
      ds[i] = tb[m.to.dsigma + i];
      t0T[i] = tb[m.to.t0 + i];
      sh[i] = tb[m.to.sigmah + i];
      rd[i] = tb[m.to.rdsig + i];
      t01[i] = tb[m.to.t01s2 + i];
      tkpT[i] = tb[m.to.tkp + i];
    }
  }
  __syncthreads();
  const int c = blockIdx.x * kBlock + threadIdx.x;
  // The planet's constants are read once, before the first store (the
  // compiler cannot prove the fields distinct from them and would reload
  // each one after every store).
  const PlanetConst& Kg = m.pc[slot];
  struct {
    float AKAP, PSURF, WW, CV, RDBRV, ADV;
  } const K = {Kg.AKAP, Kg.PSURF, Kg.WW, Kg.CV, Kg.RDBRV, Kg.ADV};
  const size_t SN = (size_t)d.S * d.NHOR;
  const FieldPtrs& F = m.f;
  const float rcsq = m.sh.rcsq[c % d.NHOR];
  // gp = exp(gp) is stored with the first tendencies below, after every
  // load: a store here would hold back the loads that follow it.
  const float ps = expf(F.gp[c]);
  const float gpm = F.gpmt[c], gpj = F.gpj[c];
  float gu[NL], gv[NL], gt[NL], gd[NL], gz[NL], gq[NL], zvgpg[NL], ztv1[NL], ztv2[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    const size_t at = l * SN + c;
    gu[l] = F.gu[at];
    gv[l] = F.gv[at];
    gt[l] = F.gt[at];
    gd[l] = F.gd[at];
    gz[l] = F.gz[at];
    gq[l] = F.gq[at];
    zvgpg[l] = rcsq * (gu[l] * gpm + gv[l] * gpj);
    const float zq = fmaxf(gq[l] / ps, 0.f);
    const float t0 = t0T[l];
    const float tvirt = (gt[l] + t0) * (1.f + (1.f / K.RDBRV - 1.f) * zq);
    ztv1[l] = tvirt - t0;
    ztv2[l] = tvirt / (1.f + K.ADV * zq) - t0;
  }
  float zsdotp[NL];
  float zsumd = ds[0] * gd[0];
  float gvp = ds[0] * zvgpg[0];
  zsdotp[0] = zsumd + gvp;
#pragma unroll
  for (int l = 1; l < NL - 1; ++l) {
    zsumd = zsumd + ds[l] * gd[l];
    gvp = gvp + ds[l] * zvgpg[l];
    zsdotp[l] = zsumd + gvp;
  }
  zsumd = zsumd + ds[NL - 1] * gd[NL - 1];
  gvp = gvp + ds[NL - 1] * zvgpg[NL - 1];
  float gtd[NL], gqm[NL], gud[NL], gvd[NL];
#pragma unroll
  for (int l = 0; l < NL - 1; ++l) {
    zsdotp[l] = sh[l] * (zsumd + gvp) - zsdotp[l];
    gtd[l] = zsdotp[l] * (gt[l + 1] - gt[l]);
    gqm[l] = zsdotp[l] * (gq[l + 1] + gq[l]);
    gud[l] = zsdotp[l] * (gu[l + 1] - gu[l]);
    gvd[l] = zsdotp[l] * (gv[l + 1] - gv[l]);
  }
  // Level tendencies go out as soon as they are formed (fewer live arrays).
  zsumd = zvgpg[0] * ds[0];
  const float rdsig0 = rd[0];
  F.gp[c] = ps;
  F.gtn[c] = gt[0] * gd[0] - K.AKAP * ztv2[0] * gd[0] - rdsig0 * (gtd[0] + t01[0] * (sh[0] * gvp - zsumd));
  F.gqn[c] = -rdsig0 * gqm[0];
  F.guz[c] = -gu[0] * gz[0] - gpj * ztv1[0] - rdsig0 * gvd[0];
  F.gvz[c] = gv[0] * gz[0] - gpm * ztv1[0] - rdsig0 * gud[0];
  F.dw[c] = gd[0] * ps * K.PSURF * K.WW;
#pragma unroll
  for (int l = 1; l < NL; ++l) {
    const int column = l * NL;
    float ztpta = C[column] * zvgpg[0];
    float ztptb = C[column] * (zvgpg[0] + gd[0]);
#pragma unroll
    for (int j = 1; j <= l; ++j) {
      ztpta = ztpta + C[column + j] * zvgpg[j];
      ztptb = ztptb + C[column + j] * (zvgpg[j] + gd[j]);
    }
    const float rdsig = rd[l], t01s2 = t01[l], t01s2m = t01[l - 1], sigmah = sh[l], sigmahm = sh[l - 1];
    const float tkp = tkpT[l];
    const size_t at = l * SN + c;
    if (l < NL - 1) {
      zsumd = zsumd + zvgpg[l] * ds[l];
      F.gtn[at] = gt[l] * gd[l] + K.AKAP * ztv2[l] * (zvgpg[l] - ztptb) + tkp * (zvgpg[l] - ztpta) -
               rdsig * (gtd[l] + gtd[l - 1] + gvp * (t01s2 * sigmah + t01s2m * sigmahm) - zsumd * (t01s2m + t01s2) +
                        zvgpg[l] * ds[l] * t01s2m);
      F.gqn[at] = -rdsig * (gqm[l] - gqm[l - 1]);
      F.guz[at] = -gu[l] * gz[l] - gpj * ztv1[l] - rdsig * (gvd[l] + gvd[l - 1]);
      F.gvz[at] = gv[l] * gz[l] - gpm * ztv1[l] - rdsig * (gud[l] + gud[l - 1]);
    } else {
      F.gtn[at] = gt[l] * gd[l] + K.AKAP * ztv2[l] * (zvgpg[l] - ztptb) + tkp * (zvgpg[l] - ztpta) -
               rdsig * (gtd[NL - 2] + t01s2m * (sigmahm * gvp - zsumd));
      F.gqn[at] = rdsig * gqm[NL - 2];
      F.guz[at] = -gu[l] * gz[l] - gpj * ztv1[l] - rdsig * gvd[NL - 2];
      F.gvz[at] = gv[l] * gz[l] - gpm * ztv1[l] - rdsig * gud[NL - 2];
    }
    F.dw[at] = (zvgpg[l] - ztptb) * ps * K.PSURF * K.WW;
  }
  const float scale = sqrtf(rcsq);
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    float gsum = 0.f;
#pragma unroll
    for (int k = 0; k < NL; ++k) gsum = gsum + G[l * NL + k] * (ztv1[k] - gt[k]);
    const float gphi = gsum * 2.f / rcsq;
    const size_t at = l * SN + c;
    F.gut[at] = gu[l] * gt[l];
    F.gvt[at] = gv[l] * gt[l];
    F.gke[at] = gu[l] * gu[l] + gv[l] * gv[l] + gphi;
    F.guq[at] = gu[l] * gq[l];
    F.gvq[at] = gv[l] * gq[l];
    F.du0[at] = K.CV * gu[l] * scale;
    F.dv0[at] = K.CV * gv[l] * scale;
  }
  F.gvpp[c] = gvp;
  F.dp0[c] = K.PSURF * ps;
}

// spectrala (dynamics/wgsl/spectrala.wgsl): the Hoskins-Simmons semi-implicit
// scheme with this slot's bm1 for its phase. A block takes 32 real
// coefficients, a thread per (coefficient, level): what couples the levels -
// the g, bm1 and tau products - reads the other levels' values from shared
// memory and sums them in level order. One thread per coefficient gathered
// NL^2 values of bm1 by itself with the level columns in 168 registers: one
// T42 planet's 15 blocks waited for those loads (10 us), 128 planets' ran at
// three blocks per SM.
constexpr int kSpecCols = 32;

template <int NL>
__global__ void __launch_bounds__(kSpecCols* NL) k_spectrala(Model m) {
  __shared__ float s_stt[NL][kSpecCols], s_atm[NL][kSpecCols], s_adt[NL][kSpecCols], s_adm[NL][kSpecCols];
  __shared__ float s_zz[NL][kSpecCols], s_sdt[NL][kSpecCols];
  pdl_wait();
  pdl_release();
  const Dims& d = m.d;
  const int lane = threadIdx.x % kSpecCols, l = threadIdx.x / kSpecCols;
  const int c = blockIdx.x * kSpecCols + lane;
  const bool inside = c < d.S * d.NRSP;
  const int slot = inside ? c / d.NRSP : 0, s = inside ? c % d.NRSP : 0;
  const StepParams& P = m.params[slot];
  const bool run = inside && P.active;
  const PlanetConst& K = m.pc[slot];
  const float* tb = slot_tabs(m, slot);
  const size_t SR = (size_t)d.S * d.NRSP, at = l * SR + c;
  const FieldPtrs& F = m.f;
  const bool filter = P.filter != 0.f;
  const float DELT = P.delt, DELT2 = P.delt2;
  float adm = 0.f, azm = 0.f, atm = 0.f, aqm = 0.f, adt = 0.f, stt = 0.f, szt = 0.f, sqt = 0.f;
  float sdp0 = 0.f, szp0 = 0.f, stp0 = 0.f, sqp0 = 0.f, apm = 0.f, spt = 0.f, spp = 0.f;
  if (run) {
    adm = F.sdm[at];
    azm = F.szm[at];
    atm = F.stm[at];
    aqm = F.sqm[at];
    adt = F.sdt[at];
    stt = F.stt[at];
    szt = F.szt[at];
    sqt = F.sqt[at];
    if (filter) {
      sdp0 = F.sdp[at];
      szp0 = F.szp[at];
      stp0 = F.stp[at];
      sqp0 = F.sqp[at];
    }
    apm = F.spm[c];
    spt = F.spt[c];
    if (l == 0) spp = F.spp[c];
  }
  s_stt[l][lane] = stt;
  s_atm[l][lane] = atm;
  s_adt[l][lane] = adt;
  s_adm[l][lane] = adm;
  __syncthreads();
  const int jn = run ? (int)m.sh.nindex[s] : 0;
  float zz = 0.f;
  if (run) {
    const float* G = tb + m.to.g + l * NL;
    float zgt = 0.f, zgm = 0.f;
#pragma unroll
    for (int k = 0; k < NL; ++k) {
      zgt = zgt + G[k] * s_stt[k][lane];
      zgm = zgm + G[k] * s_atm[k][lane];
    }
    if (jn > 0) {
      const float zq = 1.f / (float)(jn * (jn + 1));
      const float z0 = tb[m.to.t0 + l];
      const float zt = zgt - z0 * spt;
      const float zm = zgm + z0 * apm;
      const float za = adt * zq + tb[m.to.sop + s];
      const float zb = adm * zq;
      zz = zb + DELT * (zm + za + DELT * zt);
    }
  }
  s_zz[l][lane] = zz;
  __syncthreads();
  float sdt = 0.f;
  if (run && jn > 0 && s >= 2) {
    const float* bm1 = tb + m.to.bm1 + (size_t)P.phase * d.T * NL * NL + ((jn - 1) * NL + l) * NL;
    if constexpr (NL % 2 == 0) {  // every table before bm1 holds an even count then: rows start 8-byte aligned
      float2 b[NL / 2];
#pragma unroll
      for (int k = 0; k < NL / 2; ++k) b[k] = __ldg(reinterpret_cast<const float2*>(bm1) + k);
#pragma unroll
      for (int k = 0; k < NL / 2; ++k) {
        sdt = sdt + s_zz[2 * k][lane] * b[k].x;
        sdt = sdt + s_zz[2 * k + 1][lane] * b[k].y;
      }
    } else {
#pragma unroll
      for (int k = 0; k < NL; ++k) sdt = sdt + s_zz[k][lane] * __ldg(bm1 + k);
    }
  }
  s_sdt[l][lane] = sdt;
  __syncthreads();
  if (!run) return;
  {
    const float* tau = tb + m.to.tau + l * NL;
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < NL; ++k) t = t + tau[k] * s_sdt[k][lane];
    stt = stt - t;
  }
  if (l == 0) {
    const float* ds = tb + m.to.dsigma;
#pragma unroll
    for (int k = 0; k < NL; ++k) spt = spt + ds[k] * s_sdt[k][lane];
    if (filter) F.spm[c] = K.PNU21 * spp + K.PNU * apm;
    const float sppNew = s < 2 ? 0.f : apm - DELT2 * spt;
    F.spp[c] = sppNew;
    F.sp[c] = sppNew;
    F.spt[c] = spt;
  }
  const float PNU21 = K.PNU21, PNU = K.PNU;
  if (filter) {
    F.sdm[at] = __fmaf_rn(PNU21, sdp0, PNU * adm);
    F.szm[at] = __fmaf_rn(PNU21, szp0, PNU * azm);
    F.stm[at] = __fmaf_rn(PNU21, stp0, PNU * atm);
    F.sqm[at] = __fmaf_rn(PNU21, sqp0, PNU * aqm);
  }
  const float sdp = 2.f * sdt - adm;
  const float stp = DELT2 * stt + atm;
  const float szp = DELT2 * szt + azm;
  const float sqp = DELT2 * sqt + aqm;
  F.sdt[at] = sdt;
  F.stt[at] = stt;
  F.sdp[at] = sdp;
  F.stp[at] = stp;
  F.szp[at] = szp;
  F.sqp[at] = sqp;
  F.sd[at] = sdp;
  F.st[at] = stp;
  F.sz[at] = szp;
  F.sq[at] = sqp;
}

__device__ __forceinline__ float2 ld2(const float* p, size_t i) { return *reinterpret_cast<const float2*>(p + i); }
__device__ __forceinline__ void st2(float* p, size_t i, float2 v) { *reinterpret_cast<float2*>(p + i) = v; }

// spectrald up to mkdheat (dynamics/wgsl/spectrald-diffusion.wgsl). A thread
// owns two adjacent real coefficients (NRSP is even, so both are of one
// slot) of one level. Every input is read before the slot's parameters are
// tested and before the first store: the fields are distinct arrays, but
// the compiler cannot prove it, and would otherwise order each load after
// the stores before it.
__global__ void __launch_bounds__(kBlock) k_spectrald_diffusion(Model m) {
  pdl_wait();
  pdl_release();
  const Dims& d = m.d;
  const int c = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (c >= d.S * d.NRSP) return;
  const int l = blockIdx.y;
  const int slot = c / d.NRSP, s = c - slot * d.NRSP;
  const float* tb = slot_tabs(m, slot);
  const size_t at = (size_t)l * d.S * d.NRSP + c;
  const FieldPtrs& F = m.f;
  const float2 szp0 = ld2(F.szp, at), szt0 = ld2(F.szt, at), stp0 = ld2(F.stp, at), stt0 = ld2(F.stt, at);
  const float2 sdp0 = ld2(F.sdp, at), sdt0 = ld2(F.sdt, at), sqp0 = ld2(F.sqp, at), sqt0 = ld2(F.sqt, at);
  const float* sak = tb + m.to.sakpp + l * d.NRSP + s;
  const float* srpl = tb + m.to.srp + l * d.NRSP + s;
  const float sakpp[2] = {sak[0], sak[1]}, srp[2] = {srpl[0], srpl[1]};
  const float damp = tb[m.to.damp + l], tdisst = tb[m.to.tdisst + l], tdissq = tb[m.to.tdissq + l];
  const float tdissd = tb[m.to.tdissd + l], tdissz = tb[m.to.tdissz + l], tfrc = tb[m.to.tfrc + l];
  const StepParams& P = m.params[slot];
  if (!P.active) return;
  const float D2 = P.delt2, PLAVOR = m.pc[slot].PLAVOR;
  float o[12][2];  // szp, stp, sdp, sqp, stt, sqt, sdt, szt, zdsdp1, zdszp1, zdsdp2, zdszp2
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float szp = (k ? szp0.y : szp0.x) + D2 * (k ? szt0.y : szt0.x);
    const float stp = (k ? stp0.y : stp0.x) + D2 * (k ? stt0.y : stt0.x);
    const float sdp = (k ? sdp0.y : sdp0.x) + D2 * (k ? sdt0.y : sdt0.x);
    const float sqp = (k ? sqp0.y : sqp0.x) + D2 * (k ? sqt0.y : sqt0.x);
    // IEEE divisions (the file otherwise divides to 2 ulp): the diffusion
    // and friction increments feed mkdheat's heating through two more
    // transforms, where 2-ulp quotients left V3's bound. Most levels have no
    // friction and most wavenumbers no diffusion: their numerators are zero.
    const float sk = sakpp[k];
    const float stt = quotient((-damp - tdisst * sk) * stp + damp * srp[k], 1.f + D2 * (damp + tdisst * sk));
    const float sqt = quotient(-tdissq * sk * sqp, 1.f + D2 * tdissq * sk);
    const float zsdt1 = quotient(-tfrc * sdp, 1.f + D2 * tfrc);
    const float zsdt2 = quotient(-tdissd * sk * sdp, 1.f + D2 * tdissd * sk);
    float zszt1 = quotient(-tfrc * szp, 1.f + D2 * tfrc);
    float zszt2 = quotient(-tdissz * sk * szp, 1.f + D2 * tdissz * sk);
    float szt = zszt1 + zszt2;
    if (s + k == 2) {
      zszt1 = zszt1 + __fdiv_rn(PLAVOR * tfrc, 1.f + D2 * tfrc);
      zszt2 = zszt2 + __fdiv_rn(PLAVOR * tdissz * sk, 1.f + D2 * tdissz * sk);
      szt = szt + PLAVOR * (__fdiv_rn(tfrc, 1.f + D2 * tfrc) + __fdiv_rn(tdissz * sk, 1.f + D2 * tdissz * sk));
    }
    const float v[12] = {szp, stp, sdp, sqp, stt, sqt, zsdt1 + zsdt2, szt, zsdt1 * D2, zszt1 * D2, zsdt2 * D2,
                         zszt2 * D2};
#pragma unroll
    for (int j = 0; j < 12; ++j) o[j][k] = v[j];
  }
  if (l == 0 && s < 2) st2(F.spp, c, make_float2(0.f, 0.f));
  float* const dst[12] = {F.szp, F.stp, F.sdp, F.sqp, F.stt, F.sqt, F.sdt, F.szt, F.zdsdp1, F.zdszp1, F.zdsdp2, F.zdszp2};
#pragma unroll
  for (int j = 0; j < 12; ++j) st2(dst[j], at, make_float2(o[j][0], o[j][1]));
}

// Elementwise grid-point kernels give each thread four adjacent columns of
// one level (16-byte loads and stores): a block covers kCols4 = 512
// columns, and 512 divides NHOR (2048, 8192, 18432), so a block's columns
// share one slot. Four columns per thread keep four times the bytes in
// flight for the same number of resident warps.
constexpr int kCols4 = 4 * kBlock;

__device__ __forceinline__ float4 ld4(const float* p, size_t i) { return *reinterpret_cast<const float4*>(p + i); }
__device__ __forceinline__ void st4(float* p, size_t i, float4 v) { *reinterpret_cast<float4*>(p + i) = v; }

// mkdheat's first two grid-point stages (dynamics/wgsl/mkdheat.wgsl): the
// heating by friction's wind increments (zdu1, zdv1) and the kinetic energy
// the diffusion's (zdu, zdv) take, in one pass over the winds both read.
__global__ void __launch_bounds__(kBlock) k_mkdheat_winds(Model m) {
  pdl_wait();
  pdl_release();
  const Dims& d = m.d;
  const int slot = blockIdx.x * kCols4 / d.NHOR;
  const int c = blockIdx.x * kCols4 + 4 * threadIdx.x;
  const int l = blockIdx.y;
  const size_t i = (size_t)l * d.S * d.NHOR + c;
  const int h = c - slot * d.NHOR;
  const FieldPtrs& F = m.f;
  // inputs first, then the slot's parameters
  const float4 dq = ld4(F.dq, i), dp = ld4(F.dp, c);
  const float4 zu = ld4(F.zu, i), zv = ld4(F.zv, i);
  const float4 du1 = ld4(m.zdu1, i), dv1 = ld4(m.zdv1, i), du2 = ld4(F.zdu, i), dv2 = ld4(F.zdv, i);
  const float4 rc = ld4(m.sh.rcsq, h);
  const float ds = m.tabs[(size_t)slot * m.to.stride + m.to.dsigma + l];
  const StepParams& P = m.params[slot];
  if (!P.active) return;
  const PlanetConst& K = m.pc[slot];
  const float4 heat = make_float4(1.f + K.ADV * dq.x, 1.f + K.ADV * dq.y, 1.f + K.ADV * dq.z, 1.f + K.ADV * dq.w);
  auto change = [&](float r, float zu1, float zv1, float zdu1, float zdv1) {
    const float scale = K.CV * sqrtf(r);
    const float u = zu1 * scale, v = zv1 * scale, du = zdu1 * scale, dv = zdv1 * scale;
    return du * (2.f * u + du) + dv * (2.f * v + dv);
  };
  // IEEE divisions throughout mkdheat, as in spectrald's diffusion.
  auto friction = [&](float change, float ht) {
    // friction acts on the top levels alone, and an IEEE division of zero takes
    // the slow path of its routine: 128 T42 L10 planets 95 -> 58 us, as long as
    // its loads and stores take
    if (change == 0.f && isfinite(ht) && ht != 0.f) return -change * ht;
    const float dtdt = __fdiv_rn(__fdiv_rn(__fdiv_rn(-change, P.deltsec2) * 0.5f, K.ACPD), ht);
    return __fdiv_rn(__fdiv_rn(dtdt, K.CT), K.WW);
  };
  auto diffusion = [&](float change, float p) { return __fdiv_rn(__fdiv_rn(change, P.deltsec2) * p, K.GA) * ds; };
  st4(F.zdtdt, i, make_float4(friction(change(rc.x, zu.x, zv.x, du1.x, dv1.x), heat.x),
                              friction(change(rc.y, zu.y, zv.y, du1.y, dv1.y), heat.y),
                              friction(change(rc.z, zu.z, zv.z, du1.z, dv1.z), heat.z),
                              friction(change(rc.w, zu.w, zv.w, du1.w, dv1.w), heat.w)));
  st4(F.zdekin, i, make_float4(diffusion(change(rc.x, zu.x, zv.x, du2.x, dv2.x), dp.x),
                               diffusion(change(rc.y, zu.y, zv.y, du2.y, dv2.y), dp.y),
                               diffusion(change(rc.z, zu.z, zv.z, du2.z, dv2.z), dp.z),
                               diffusion(change(rc.w, zu.w, zv.w, du2.w, dv2.w), dp.w)));
}

// mkdheat's third stage. Between the second and the third the shaders
// transform the kinetic energy to spectral space, keep mode (0, 0) alone
// (dynamics/wgsl/mean-mode.wgsl) and transform that back. Only fc2sp's sum
// of mode (0, 0) reaches the result, over the latitude pairs of the Fourier
// rows' mean (m = 0, in the scratch fzdv1), and back on the grid a latitude is
// the constant q(0, 0)[lat] times it, exactly: every other term of sp2fc and
// fc2gp is a sum with zeros. So each block takes that sum in the shaders'
// order and no transform runs (fc2sp, the zeroing, sp2gp and this stage's
// read of zdekin took 20 + 8 + 33 + 8 us at 128 T42 L10 planets, and three
// of a single planet's launches). The slot's first block also writes the
// spectral field, and with `fourier` the slot's blocks the Fourier field
// between the two (a row's m = 0 is that constant, the rest zero). A block
// takes `chunks` runs of kCols4 columns of its plane, so that the sum, a chain
// of NLAT / 2 multiply-adds in one warp, is taken once for all of them.
__global__ void __launch_bounds__(kBlock) k_mkdheat_mean(Model m, int chunks, int fourier) {
  constexpr int kMaxPairs = 48;
  __shared__ float pair_sum[kMaxPairs], pair_q[kMaxPairs];
  __shared__ float mean;
  pdl_wait();
  pdl_release();
  const Dims& d = m.d;
  const int first = blockIdx.x * chunks * kCols4;  // the block's columns, all of one slot
  const int slot = first / d.NHOR;
  const int l = blockIdx.y;
  const FieldPtrs& F = m.f;
  const size_t plane = (size_t)l * d.S + slot;
  if (threadIdx.x < 32) {
    const float* rows = m.fzdv1 + plane * d.NLAT * d.NFC;
    const int step = m.mode >= 1 ? 2 : d.NFC;  // m-major or latitude-major
    const int half = d.NLAT / 2;
    for (int j = threadIdx.x; j < half; j += 32) {
      pair_sum[j] = rows[j * step] + rows[(d.NLAT - 1 - j) * step];
      pair_q[j] = m.sh.qc[(size_t)j * d.NCSP];
    }
    __syncwarp();
    float s = 0.f;
#pragma unroll 4
    for (int j = 0; j < half; ++j) s = fmaf(pair_q[j], pair_sum[j], s);
    if (threadIdx.x == 0) mean = s;
  }
  const float ds = m.tabs[(size_t)slot * m.to.stride + m.to.dsigma + l];
  const StepParams& P = m.params[slot];
  __syncthreads();
  if (!P.active) return;
  const PlanetConst& K = m.pc[slot];
  const float s00 = mean;
  if (first == slot * d.NHOR) {
    float* out = F.zsdef + plane * d.NRSP;
    for (int r = threadIdx.x; r < d.NRSP; r += kBlock) out[r] = r == 0 ? s00 : 0.f;
  }
  if (fourier) {
    float* out = F.fzdekin + plane * d.NLAT * d.NFC;
    const int block = (first - slot * d.NHOR) / (chunks * kCols4), blocks = d.NHOR / (chunks * kCols4);
    for (int i = block * kBlock + threadIdx.x; i < d.NLAT * d.NFC; i += blocks * kBlock) {
      const bool mean_part = m.mode >= 1 ? i < 2 * d.NLAT && i % 2 == 0 : i % d.NFC == 0;  // m-major or latitude-major
      const int lat = m.mode >= 1 ? i / 2 : i / d.NFC;
      out[i] = mean_part ? m.sh.qi[(size_t)lat * d.NCSP] * s00 : 0.f;
    }
  }
  for (int k = 0; k < chunks; ++k) {
    const int c = first + k * kCols4 + 4 * threadIdx.x;
    const size_t i = (size_t)l * d.S * d.NHOR + c;
    const float4 dq = ld4(F.dq, i), dp = ld4(F.dp, c);
    const float ek = m.sh.qi[(size_t)((c - slot * d.NHOR) / d.NLON) * d.NCSP] * s00;
    st4(F.zdekin, i, make_float4(ek, ek, ek, ek));
    const float4 heat = make_float4(1.f + K.ADV * dq.x, 1.f + K.ADV * dq.y, 1.f + K.ADV * dq.z, 1.f + K.ADV * dq.w);
    // IEEE divisions, as above.
    auto one = [&](float ht, float p) {
      const float dtdt = __fdiv_rn(__fdiv_rn(__fdiv_rn(__fdiv_rn(-ek * 0.5f, K.ACPD), ht), p) * K.GA, ds);
      return __fdiv_rn(__fdiv_rn(dtdt, K.CT), K.WW);
    };
    st4(F.zdtdt, i, make_float4(one(heat.x, dp.x), one(heat.y, dp.y), one(heat.z, dp.z), one(heat.w, dp.w)));
  }
}

// spectrald after mkdheat (dynamics/wgsl/spectrald-update.wgsl), two
// adjacent real coefficients of one level per thread, inputs read first.
__global__ void __launch_bounds__(kBlock) k_spectrald_update(Model m) {
  pdl_wait();
  pdl_release();
  const Dims& d = m.d;
  const int c = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (c >= d.S * d.NRSP) return;
  const int l = blockIdx.y;
  const int slot = c / d.NRSP;
  const size_t at = (size_t)l * d.S * d.NRSP + c;
  const FieldPtrs& F = m.f;
  const float2 stt0 = ld2(F.stt, at), zstt1 = ld2(F.zstt1, at), zstt2 = ld2(F.zstt2, at);
  const float2 szp0 = ld2(F.szp, at), szt = ld2(F.szt, at), stp0 = ld2(F.stp, at), sdp0 = ld2(F.sdp, at);
  const float2 sdt = ld2(F.sdt, at), sqp0 = ld2(F.sqp, at), sqt = ld2(F.sqt, at);
  const bool surface = l == 0;  // the level-0 threads also update sp
  const float2 spp = surface ? ld2(F.spp, c) : make_float2(0.f, 0.f);
  const StepParams& P = m.params[slot];
  if (!P.active) return;
  const float PNU = m.pc[slot].PNU;
  const bool filter = P.filter != 0.f;
  const float D2 = P.delt2;
  float2 szm = make_float2(0.f, 0.f), stm = szm, sdm = szm, sqm = szm, spm = szm;
  if (filter) {
    szm = ld2(F.szm, at);
    stm = ld2(F.stm, at);
    sdm = ld2(F.sdm, at);
    sqm = ld2(F.sqm, at);
    if (surface) spm = ld2(F.spm, c);
  }
  const float2 stt = make_float2(stt0.x + zstt1.x + zstt2.x, stt0.y + zstt1.y + zstt2.y);
  const float2 szp = make_float2(szp0.x + D2 * szt.x, szp0.y + D2 * szt.y);
  const float2 stp = make_float2(stp0.x + D2 * stt.x, stp0.y + D2 * stt.y);
  const float2 sdp = make_float2(sdp0.x + D2 * sdt.x, sdp0.y + D2 * sdt.y);
  const float2 sqp = make_float2(sqp0.x + D2 * sqt.x, sqp0.y + D2 * sqt.y);
  if (surface) {
    if (filter) st2(F.spm, c, make_float2(spm.x + PNU * spp.x, spm.y + PNU * spp.y));
    st2(F.sp, c, spp);
  }
  st2(F.stt, at, stt);
  st2(F.szp, at, szp);
  st2(F.stp, at, stp);
  st2(F.sdp, at, sdp);
  st2(F.sqp, at, sqp);
  if (filter) {
    st2(F.szm, at, make_float2(szm.x + PNU * szp.x, szm.y + PNU * szp.y));
    st2(F.stm, at, make_float2(stm.x + PNU * stp.x, stm.y + PNU * stp.y));
    st2(F.sdm, at, make_float2(sdm.x + PNU * sdp.x, sdm.y + PNU * sdp.y));
    st2(F.sqm, at, make_float2(sqm.x + PNU * sqp.x, sqm.y + PNU * sqp.y));
  }
  st2(F.sz, at, szp);
  st2(F.st, at, stp);
  st2(F.sd, at, sdp);
  st2(F.sq, at, sqp);
}

// gridpointd before the parameterizations (dynamics/wgsl/physics-in.wgsl),
// one thread per column, every input read before the first store. A block's
// columns share one slot: kBlock divides NHOR. The grid tendencies, and the
// dimensional ones below the surface level, are zeroed only under
// single-stage replay (Model::zero_gdt); within a full step the fixer's column
// stage follows here, from the humidity in registers (a kernel of its own read
// it back: 15 us at 128 T42 L10 planets, and a launch).
template <int NL>
__global__ void __launch_bounds__(kBlock) k_physics_in(Model m) {
  pdl_wait();
  pdl_release();
  const Dims& d = m.d;
  const int slot = blockIdx.x * kBlock / d.NHOR;
  if (!m.params[slot].active) return;
  const int c = blockIdx.x * kBlock + threadIdx.x;
  const int h = c - slot * d.NHOR;
  const PlanetConst& K = m.pc[slot];
  const float PSURF = K.PSURF, CV = K.CV, CT = K.CT;
  const float* t0 = m.tabs + (size_t)slot * m.to.stride + m.to.t0;
  const size_t SN = (size_t)d.S * d.NHOR;
  const FieldPtrs& F = m.f;
  const float gp = F.gp[c], rcsq = m.sh.rcsq[h];
  float gu[NL], gv[NL], gt[NL], gq[NL], t0l[NL], dsl[NL], dq[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    const size_t at = l * SN + c;
    gu[l] = F.gu[at];
    gv[l] = F.gv[at];
    gt[l] = F.gt[at];
    gq[l] = F.gq[at];
    t0l[l] = t0[l];
    dsl[l] = m.tabs[(size_t)slot * m.to.stride + m.to.dsigma + l];
  }
  const float dp = PSURF * expf(gp);
  F.dp[c] = dp;
  const float scale = sqrtf(rcsq);
#pragma unroll
  for (int l = 0; l < NL + 1; ++l) {
    const size_t at = l * SN + c;
    if (m.zero_gdt || l == NL) {
      F.dudt[at] = 0.f;
      F.dvdt[at] = 0.f;
      F.dtdt[at] = 0.f;
      F.dqdt[at] = 0.f;
    }
    if (l < NL) {
      if (m.zero_gdt) {
        F.gudt[at] = 0.f;
        F.gvdt[at] = 0.f;
        F.gtdt[at] = 0.f;
        F.gqdt[at] = 0.f;
      }
      F.du[at] = CV * gu[l] * scale;
      F.dv[at] = CV * gv[l] * scale;
      F.dt[at] = CT * (gt[l] + t0l[l]);
      dq[l] = gq[l] * PSURF / dp;
      F.dq[at] = dq[l];
    }
  }
  if (!m.zero_gdt) fixer_column<NL>(m, dsl, SN, c, h, dq, dp);
}

// gridpointd after the parameterizations (dynamics/wgsl/physics-out.wgsl),
// four columns of one level per thread, inputs read before the stores.
// Within a full step gudt, gvdt, gtdt hold no earlier increment and are not
// read (Model::zero_gdt): the sum adds +0 as the zeroed fields would.
__global__ void __launch_bounds__(kBlock) k_physics_out(Model m) {
  pdl_wait();
  pdl_release();
  const Dims& d = m.d;
  const int slot = blockIdx.x * kCols4 / d.NHOR;
  const int c = blockIdx.x * kCols4 + 4 * threadIdx.x;
  const int h = c - slot * d.NHOR;
  const size_t i = (size_t)blockIdx.y * d.S * d.NHOR + c;
  const FieldPtrs& F = m.f;
  const float4 dudt = ld4(F.dudt, i), dvdt = ld4(F.dvdt, i), dtdt = ld4(F.dtdt, i), dqdt = ld4(F.dqdt, i);
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool earlier = m.zero_gdt != 0;
  const float4 gudt = earlier ? ld4(F.gudt, i) : z, gvdt = earlier ? ld4(F.gvdt, i) : z;
  const float4 gtdt = earlier ? ld4(F.gtdt, i) : z, gqdt = ld4(F.gqdt, i);
  const float4 dp = ld4(F.dp, c), rc = ld4(m.sh.rcsq, h);
  if (!m.params[slot].active) return;
  const PlanetConst& K = m.pc[slot];
  const float CV = K.CV, WW = K.WW, CT = K.CT, PSURF = K.PSURF;
  const float4 scale = make_float4(sqrtf(rc.x), sqrtf(rc.y), sqrtf(rc.z), sqrtf(rc.w));
  auto wind = [&](float4 t, float4 g) {
    return make_float4(t.x / scale.x / CV / WW + g.x, t.y / scale.y / CV / WW + g.y, t.z / scale.z / CV / WW + g.z,
                       t.w / scale.w / CV / WW + g.w);
  };
  st4(F.gudt, i, wind(dudt, gudt));
  st4(F.gvdt, i, wind(dvdt, gvdt));
  st4(F.gtdt, i, make_float4(dtdt.x / CT / WW + gtdt.x, dtdt.y / CT / WW + gtdt.y, dtdt.z / CT / WW + gtdt.z,
                             dtdt.w / CT / WW + gtdt.w));
  st4(F.gqdt, i, make_float4(dqdt.x * dp.x / WW / PSURF + gqdt.x, dqdt.y * dp.y / WW / PSURF + gqdt.y,
                             dqdt.z * dp.z / WW / PSURF + gqdt.z, dqdt.w * dp.w / WW / PSURF + gqdt.w));
}

inline unsigned blocks(size_t n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

void dyn_calcgp(const Model& m, cudaStream_t st) {
  static_assert(2048 % kBlock == 0, "k_calcgp assumes a block lies in one slot");
  const unsigned n = (unsigned)((size_t)m.d.S * m.d.NHOR / kBlock);
  if (m.d.L == 10)
    step_launch(m.pdl, k_calcgp<10>, n, kBlock, 0, st, m);
  else
    step_launch(m.pdl, k_calcgp<5>, n, kBlock, 0, st, m);
}
void dyn_spectrala(const Model& m, cudaStream_t st) {
  const unsigned n = blocks((size_t)m.d.S * m.d.NRSP, kSpecCols);
  if (m.d.L == 10)
    step_launch(m.pdl, k_spectrala<10>, n, kSpecCols * 10, 0, st, m);
  else
    step_launch(m.pdl, k_spectrala<5>, n, kSpecCols * 5, 0, st, m);
}
void dyn_spectrald_diffusion(const Model& m, cudaStream_t st) {
  const dim3 grid(blocks((size_t)m.d.S * m.d.NRSP / 2, kBlock), m.d.NLEV);
  step_launch(m.pdl, k_spectrald_diffusion, grid, kBlock, 0, st, m);
}
void dyn_mkdheat_winds(const Model& m, cudaStream_t st) {
  const dim3 grid((unsigned)((size_t)m.d.S * m.d.NHOR / kCols4), m.d.NLEV);
  step_launch(m.pdl, k_mkdheat_winds, grid, kBlock, 0, st, m);
}
void dyn_mkdheat_mean(const Model& m, cudaStream_t st) {
  // 4 kCols4 = 2,048 divides NHOR; four runs a block once that leaves several
  // blocks per SM
  const size_t runs = (size_t)m.d.S * m.d.NHOR / kCols4;
  const int chunks = runs * m.d.NLEV >= (size_t)sm_count() * 32 ? 4 : 1;
  const dim3 grid((unsigned)(runs / chunks), m.d.NLEV);
  // mode 1 leaves the Fourier fields between fused transforms unwritten
  const int fourier = m.mode != 1 || m.keep_fourier;
  step_launch(m.pdl, k_mkdheat_mean, grid, kBlock, 0, st, m, chunks, fourier);
}
void dyn_spectrald_update(const Model& m, cudaStream_t st) {
  const dim3 grid(blocks((size_t)m.d.S * m.d.NRSP / 2, kBlock), m.d.NLEV);
  step_launch(m.pdl, k_spectrald_update, grid, kBlock, 0, st, m);
}
void dyn_physics_in(const Model& m, cudaStream_t st) {
  const unsigned n = (unsigned)((size_t)m.d.S * m.d.NHOR / kBlock);
  if (m.d.L == 10)
    step_launch(m.pdl, k_physics_in<10>, n, kBlock, 0, st, m);
  else
    step_launch(m.pdl, k_physics_in<5>, n, kBlock, 0, st, m);
}
void dyn_physics_out(const Model& m, cudaStream_t st) {
  const dim3 grid((unsigned)((size_t)m.d.S * m.d.NHOR / kCols4), m.d.NLEV);
  step_launch(m.pdl, k_physics_out, grid, kBlock, 0, st, m);
}

}  // namespace exogcm
