// Convection and rain with a thread per (column, level), for batches of few
// columns (phy_levels). A block takes 32 columns, warp l their level l:
// what a routine does for each level on its own runs on NL times the threads,
// from code that is not unrolled over the levels, and what couples the levels
// - recurrences over values already formed - is taken by one warp or by each
// level over the others, through shared memory.
//
// One thread per column (physics.cu) has the fewer
// instructions and wins where the columns fill the chip. One planet's 2,048 to
// 18,432 columns do not: they run as 16 to 144 blocks of one warp per
// scheduler, each waiting out the routine's whole chain of ten levels and the
// fetch of its code. Every value is formed by the same operations in the same
// order as there, so a planet's result does not depend on the batch it is in.
#include "physics_common.cuh"

namespace exogcm {

namespace {

constexpr int kCols = 32;  // columns of a block; kCols divides NHOR, so they are of one slot

#define LEVEL_PROLOGUE                                               \
  pdl_wait();                                                        \
  pdl_release();                                                     \
  const Dims& d = m.d;                                               \
  const int lane = threadIdx.x & 31, l = threadIdx.x >> 5;           \
  const int slot = blockIdx.x * kCols / d.NHOR;                      \
  const StepParams& P = m.params[slot];                              \
  if (!P.active) return;                                             \
  const PlanetConst& K = pcr[slot];                                  \
  const float* __restrict__ tb = tabr + (size_t)slot * m.to.stride;  \
  const int c = blockIdx.x * kCols + lane;                           \
  const size_t SN = (size_t)d.S * d.NHOR, at = l * SN + c;           \
  const FieldPtrs& F = m.f;                                          \
  (void)at;

// ---------------------------------------------------------------- rain
// k_rain_column's routine: the condensation, the saturation state and
// evaporation limits of mkrain, and the clouds are each level's own; mkrain's
// falling fluxes, the vapour column, the heights and the clear fraction run
// over the levels.
template <int NL>
__global__ void __launch_bounds__(32 * NL)
    k_rain_levels(Model m, const PlanetConst* __restrict__ pcr, const float* __restrict__ tabr) {
  __shared__ float s_cl[NL][kCols], s_scl[NL][kCols], s_ll[NL][kCols];         // mkrain's sources, then its results
  __shared__ float s_t[NL + 1][kCols], s_q[NL][kCols];                         // temperature (and the surface's), humidity
  __shared__ float s_melt[NL][kCols], s_water[NL][kCols], s_ice[NL][kCols];    // latent heats over heat capacity
  __shared__ float s_lwater[NL][kCols], s_lice[NL][kCols];                     // evaporation limits; negative: none
  __shared__ float s_zdh[NL][kCols], s_cover[NL][kCols];
  __shared__ float s_vapour[kCols], s_total[kCols], s_conv[kCols];
  LEVEL_PROLOGUE
  const float D2 = P.deltsec2;
  const bool skip = F.dca_skip[slot] != 0.f;
  const float dp = F.dp[c];
  const float dq = F.dq[at], dt = F.dt[at];
  float dtdt = F.dtdt[at], dqdt = F.dqdt[at];
  const float scl = F.dprscl[at], cl = F.dprcl[at], icclev = F.icclev[at];
  const float dw = K.CLWFAC > 0.f ? F.dw[at] : 0.f;
  const float convective = l == 0 ? F.icctot[c] : 0.f;
  const float tsurf = l == 0 ? F.dt[NL * SN + c] : 0.f;
  const float dsl = tb[m.to.dsigma + l], sgl = tb[m.to.sigma + l], lnsigl = tb[m.to.rad_lnsig + l];
  const float p = dp * sgl;
  if (!skip) {
    dtdt = dtdt + F.dca_dtdt[at];
    dqdt = dqdt + F.dca_dqdt[at];
  }
  // mklsp
  float dprll = 0.f;
  {
    const float zq = dq + dqdt * D2;
    const float zt = dt + dtdt * D2;
    const float zlcpe = __fdiv_rn(K.ALV, K.ACPD * (1.f + K.ADV * dq));
    float zqsat = sat_capped_rn(K, zt, p);
    float zcor = __fdiv_rn(1.f, 1.f - K.MOIST * zqsat);
    zqsat = zqsat * zcor;
    if (zqsat < 0.f) zqsat = 0.f;
    if (zq > zqsat) {
      float zdqdt = __fdiv_rn(zqsat - zq, 1.f + __fdiv_rn(zlcpe * K.RA2 * (K.TMELT - K.RA4) * zqsat * zcor,
                                                          (zt - K.RA4) * (zt - K.RA4)));
      float ztn = zt - zdqdt * zlcpe;
      float zqn = zq + zdqdt;
      zqsat = sat_capped_rn(K, ztn, p);
      zcor = __fdiv_rn(1.f, 1.f - K.MOIST * zqsat);
      zqsat = zqsat * zcor;
      zdqdt = __fdiv_rn(zqsat - zqn, 1.f + __fdiv_rn(zlcpe * K.RA2 * (K.TMELT - K.RA4) * zqsat * zcor,
                                                     (ztn - K.RA4) * (ztn - K.RA4)));
      ztn = ztn - zdqdt * zlcpe;
      zqn = zqn + zdqdt;
      const float lq = __fdiv_rn(zqn - zq, D2), lt = __fdiv_rn(ztn - zt, D2);
      dqdt = dqdt + lq;
      dtdt = dtdt + lt;
      dprll = -fminf(lq, 0.f) * dsl;
    }
    F.dprsll[at] = 0.f;
    F.dprll[at] = dprll;
  }
  // mkrain: what the level gives and takes of the falling fluxes
  {
    const float zq = dq + dqdt * D2;
    const float zt = dt + dtdt * D2;
    float zqsat = sat_capped(K, zt, p);
    const float zcor = 1.f / (1.f - K.MOIST * zqsat);
    zqsat = zqsat * zcor;
    if (zqsat < 0.f) zqsat = 0.f;
    const float water = K.ALV / (K.ACPD * (1.f + K.ADV * dq));
    const float ice = K.ALS / (K.ACPD * (1.f + K.ADV * dq));
    float lwater = -1.f, lice = -1.f;
    if (zq < zqsat) {
      const float deficit = zqsat - zq;
      const float curve = K.RA2 * (K.TMELT - K.RA4) * zqsat * zcor / ((zt - K.RA4) * (zt - K.RA4));
      lwater = K.GAMMA * deficit * dsl / D2 / (1.f + water * curve);
      lice = K.GAMMA * deficit * dsl / D2 / (1.f + ice * curve);
    }
    s_cl[l][lane] = cl;
    s_scl[l][lane] = scl;
    s_ll[l][lane] = dprll;
    s_t[l][lane] = dt;
    if (l == 0) s_t[NL][lane] = tsurf;
    s_q[l][lane] = dq;
    s_melt[l][lane] = (K.ALS - K.ALV) / (K.ACPD * (1.f + K.ADV * dq));
    s_water[l][lane] = water;
    s_ice[l][lane] = ice;
    s_lwater[l][lane] = lwater;
    s_lice[l][lane] = lice;
    s_zdh[l][lane] = -dt * K.GASCON / K.GA * lnsigl;
  }
  __syncthreads();
  if (l == 0) {
    const float* __restrict__ ds = tb + m.to.dsigma;
    float zprc = 0.f, zprl = 0.f, zprsc = 0.f, zprsl = 0.f;
#pragma unroll 1
    for (int k = 0; k < NL; ++k) {
      const float dsk = ds[k];
      float zdtdt = 0.f, zdqdtl = 0.f, zdqdts = 0.f;
      const float sclk = s_scl[k][lane];
      zprc = zprc + s_cl[k][lane] - sclk;
      zprl = zprl + s_ll[k][lane] - 0.f;
      zprsc = zprsc + sclk;
      zprsl = zprsl + 0.f;
      const float zlcp = s_melt[k][lane];
      const int surface = k == NL - 1 ? 2 : 1;
      for (int below = 0; below < surface; ++below) {
        const float temperature = s_t[k + below][lane];
        if (zprsc + zprsl > 0.f && temperature > K.TMELT) {
          zdtdt = -(zprsc + zprsl) / dsk * zlcp + zdtdt;
          zprc = zprsc + zprc;
          zprl = zprsl + zprl;
          zprsc = 0.f;
          zprsl = 0.f;
        } else if (zprc + zprl > 0.f && temperature <= K.TMELT) {
          zdtdt = (zprc + zprl) / dsk * zlcp + zdtdt;
          zprsc = zprc + zprsc;
          zprsl = zprl + zprsl;
          zprc = 0.f;
          zprl = 0.f;
        }
      }
      const float lwater = s_lwater[k][lane], lice = s_lice[k][lane];
      const float water = s_water[k][lane], ice = s_ice[k][lane];
      if (!(lwater == -1.f)) {
        auto evap = [&](float& flux, float limit) {
          const float zd = fminf(limit, flux);
          flux = flux - zd;
          return zd / dsk;
        };
        if (zprl > 0.f) {
          const float e = evap(zprl, lwater);
          zdtdt = zdtdt - e * water;
          zdqdtl = zdqdtl + e;
        }
        if (zprc > 0.f) {
          const float e = evap(zprc, lwater);
          zdtdt = zdtdt - e * water;
          zdqdtl = zdqdtl + e;
        }
        if (zprsl > 0.f) {
          const float e = evap(zprsl, lice);
          zdtdt = zdtdt - e * ice;
          zdqdts = zdqdts + e;
        }
        if (zprsc > 0.f) {
          const float e = evap(zprsc, lice);
          zdtdt = zdtdt - e * ice;
          zdqdts = zdqdts + e;
        }
      }
      s_cl[k][lane] = zdtdt;  // the sources are spent
      s_scl[k][lane] = zdqdtl;
      s_ll[k][lane] = zdqdts;
    }
    const float dprc = (zprc + zprsc) * dp / K.GA / 1000.f;
    F.dprc[c] = dprc;
    F.dprl[c] = (zprl + zprsl) * dp / K.GA / 1000.f;
    F.dprs[c] = (zprsc + zprsl) * dp / K.GA / 1000.f;
    const float ZCCA = 0.245f, ZCCB = 0.125f, ZCCMAX = 0.8f, ZCCMIN = 0.05f;
    float zcctot = ZCCMIN, zccconv = ZCCMIN;
    if (dprc > 0.f) {
      zcctot = ZCCA + ZCCB * logf(dprc * K.ZRFAC);
      zcctot = fminf(ZCCMAX, fmaxf(ZCCMIN, zcctot));
      zccconv = convective == 0.f ? 1.f : 1.f - fpow(1.f - zcctot, 1.f / convective);
    }
    s_total[lane] = zcctot;
    s_conv[lane] = zccconv;
  } else if (l == 1) {
    // the vapour column, beside the fluxes
    const float* __restrict__ ds = tb + m.to.dsigma;
    float dqvi = 0.f;
#pragma unroll
    for (int k = NL - 1; k >= 1; --k) dqvi = s_q[k][lane] * ds[k] + dqvi;
    dqvi = s_q[0][lane] * ds[0] + dqvi;
    dqvi = dqvi * dp / K.GA;
    F.dqvi[c] = dqvi;
    s_vapour[lane] = 700.f * logf(1.f + dqvi);
  }
  // the level's height, from the ones below it
  float zzf = 0.f;
  for (int k = NL - 1; k > l; --k) zzf = zzf + s_zdh[k][lane];
  zzf = l >= 1 ? zzf + s_zdh[l][lane] * 0.5f : zzf - dt * K.GASCON / K.GA * lnsigl;
  __syncthreads();
  dqdt = dqdt + s_scl[l][lane] + s_ll[l][lane];
  dtdt = dtdt + s_cl[l][lane];
  // mkclouds
  const float ZCLMAX = 1.f;
  float cover;
  {
    const float zcctot = s_total[lane], zccconv = s_conv[lane];
    const float zt = dt + dtdt * D2;
    const float zq = dq + dqdt * D2;
    const float zqsat = sat_divided(K, zt, p);
    float zrh = zq / zqsat;
    float dcc = icclev > 0.f ? zccconv : 0.f;
    if (icclev == 2.f && zcctot >= 0.3f) dcc = fminf(dcc + 2.f * (zcctot - 0.3f), ZCLMAX);
    zrh = zrh * (1.f - dcc);
    const float zrcrit = tb[m.to.rcrit + l];
    float zwfac = 1.f;
    if (sgl > 0.8f && K.CLWFAC > 0.f) {
      zwfac = K.CLWFAC * fmaxf(0.f, K.CLWCRIT1 - dw);
      if (K.CLWCRIT2 > dw) zwfac = 1.f;
    }
    const float excess = fmaxf(0.f, (zrh - zrcrit) / (1.f - zrcrit));
    cover = fminf(dcc + zwfac * (excess * excess), ZCLMAX);
  }
  s_cover[l][lane] = cover;
  const float zzh = s_vapour[lane];
  float dql = 0.f;
  if (zzh > 0.f && cover > 0.f) {
    dql = 0.00021f * expf(-zzf / zzh) * K.GASCON * dt / (sgl * dp);
    dql = fmaxf(dql, 1.0e-9f);
  }
  F.dql[at] = dql;
  F.dcc[at] = cover;
  F.dtdt[at] = dtdt;
  F.dqdt[at] = dqdt;
  __syncthreads();
  if (l == 0) {
    float clear = 1.f;
#pragma unroll
    for (int k = 0; k < NL - 1; ++k) clear = __fmul_rn(clear, 1.f - s_cover[k][lane]);
    F.dql[NL * SN + c] = 0.f;
    F.dcc[NL * SN + c] = __fmaf_rn(-clear, 1.f - s_cover[NL - 1][lane], 1.f);
  }
}

// ---------------------------------------------------------------- kuo
// k_kuo's routine: every level lifts its own parcel (the surface's in the
// lowest); the first level from below whose parcel is buoyant starts the
// cloud, which one warp follows up the column; the shallow convection's
// humidity and temperature are diffused by a warp each.
template <int NL>
__global__ void __launch_bounds__(32 * NL)
    k_kuo_levels(Model m, const PlanetConst* __restrict__ pcr, const float* __restrict__ tabr) {
  __shared__ float s_tot[NL][kCols], s_qe[NL][kCols], s_te[NL][kCols], s_acpe[NL][kCols], s_qsa[NL][kCols];
  __shared__ float s_pt[NL][kCols], s_pq[NL][kCols], s_pc[NL][kCols];  // each level's parcel
  __shared__ float s_dq[NL][kCols], s_dt[NL][kCols];                   // zdqdt, zdtdt
  __shared__ float s_kq[NL][kCols], s_kt[NL][kCols];
  __shared__ float s_zi[kCols], s_zat[kCols], s_zaq[kCols];
  __shared__ int s_ilift[kCols], s_itop[kCols], s_flag[NL][kCols];
  LEVEL_PROLOGUE
  constexpr int NM = NL - 1;
  const float* __restrict__ ds = tb + m.to.dsigma;
  const float* __restrict__ sg = tb + m.to.sigma;
  const float D2 = P.deltsec2;
  const float dp = F.dp[c];
  const float dqt_in = F.dqt[at], dq_in = F.dq[at], dqdt_in = F.dqdt[at], dt_in = F.dt[at], dtdt_in = F.dtdt[at];
  const float dsl = ds[l], sgl = sg[l];
  const float zdqt = dqt_in * K.PSURF * K.WW / dp;
  if (l == 0 && c == slot * d.NHOR) F.dca_skip[slot] = 0.f;  // raised again by mkdca's columns
  F.dqt[at] = zdqt;
  const float zqe = dq_in + dqdt_in * D2, zte = dt_in + dtdt_in * D2;
  const float zacpe = K.ACPD * (1.f + K.ADV * dq_in);
  s_tot[l][lane] = (zdqt + dqdt_in) * D2;
  s_qe[l][lane] = zqe;
  s_te[l][lane] = zte;
  s_acpe[l][lane] = zacpe;
  s_dq[l][lane] = 0.f;
  s_dt[l][lane] = 0.f;
  __syncthreads();
  {
    const float p = dp * sgl;
    Parcel parcel{0.f, 0.f, 0.f, false};
    bool lifts = false;
    float zqsa = 0.f;
    if (l == NM) {
      const float ztsurf = F.dt[NL * SN + c] * tb[m.to.vdiff_skap + l];
      zqsa = sat_divided(K, zte, p);
      if (s_tot[l][lane] > 0.f && ztsurf > zte) {
        const float zqnew = F.dq[NL * SN + c] * fminf(1.f, zqe / zqsa);
        parcel = condense(K, ztsurf, zqnew, p);
        lifts = parcel.saturated;
      }
    } else {
      zqsa = sat_divided(K, zte, p);
      if (s_tot[l + 1][lane] > 0.f) {
        parcel = condense(K, s_te[l + 1][lane] * tb[m.to.kuo_zfac + l], s_qe[l + 1][lane], p);
        lifts = parcel.saturated && parcel.t > zte;
      }
    }
    s_qsa[l][lane] = zqsa;
    s_pt[l][lane] = parcel.t;
    s_pq[l][lane] = parcel.q;
    s_pc[l][lane] = parcel.cor;
    s_flag[l][lane] = lifts;
  }
  __syncthreads();
  if (l == 0) {
    int ilift = -1, itop = -1;
    float zi = 0.f, zpt = 0.f, zpq = 0.f, zbeta = 0.f, zpbeta = 0.f, ztp = 0.f, zqp = 0.f;
    int from = NL - 1;
    while (from >= 0 && !s_flag[from][lane]) --from;
    if (from >= 0) {
      ztp = s_pt[from][lane];
      zqp = s_pq[from][lane];
      const float dsf = ds[from], zqsa = s_qsa[from][lane];
      ilift = from + 2;
      itop = from + 1;
      const float ddq = fmaxf(zqsa - s_qe[from][lane], 0.f), ddt = ztp - s_te[from][lane];
      s_dq[from][lane] = ddq;
      s_dt[from][lane] = ddt;
      zpt = ddt * dsf * s_acpe[from][lane];
      zpq = ddq * dsf * K.ALV;
      zbeta = fminf(1.f, s_qe[from][lane] / zqsa) * dsf;
      zpbeta = dsf;
      if (from == NM) {
        zi = s_tot[from][lane] * dsf * K.ALV;
      } else {
        const int lp = from + 1;
        const float dsp = ds[lp], pp = dp * sg[lp];
        float zqsnl = s_qsa[lp][lane];
        if (s_qe[lp][lane] > zqsnl) {
          float t = s_te[lp][lane], q = s_qe[lp][lane];
          const float lcp = (t < K.TMELT ? K.ALS : K.ALV) / (K.ACPD * (1.f + K.ADV * q));
          float cor = s_pc[from][lane];
          for (int i = 0; i < 2; ++i) {
            if (i == 1) {
              zqsnl = sat_capped(K, t, pp);
              cor = 1.f / (1.f - K.MOIST * zqsnl);
              zqsnl = zqsnl * cor;
            }
            const float dqsdt = K.RA2 * (K.TMELT - K.RA4) * zqsnl * cor / ((t - K.RA4) * (t - K.RA4));
            const float rain = (q - zqsnl) / (1.f + lcp * dqsdt);
            t = t + lcp * rain;
            q = q - rain;
          }
          const float pdq = fmaxf(q - s_qe[lp][lane], 0.f), pdt = t - s_te[lp][lane];
          s_dq[lp][lane] = pdq;
          s_dt[lp][lane] = pdt;
          zpt = pdt * dsp * s_acpe[lp][lane] + zpt;
          zpq = pdq * dsp * K.ALV + zpq;
          zbeta = fminf(1.f, s_qe[lp][lane] / zqsnl) * dsp + zbeta;
          zpbeta = dsp + zpbeta;
        }
        zi = s_tot[from][lane] * dsf * K.ALV + s_tot[lp][lane] * dsp * K.ALV;
      }
    }
#pragma unroll 1
    for (int k = from - 1; k >= 0; --k) {
      const Parcel parcel = condense(K, ztp * tb[m.to.kuo_zfac + k], zqp, dp * sg[k]);
      if (!(parcel.saturated && parcel.t > s_te[k][lane])) break;
      const float dsk = ds[k], zqsa = s_qsa[k][lane];
      itop = k + 1;
      ztp = parcel.t;
      zqp = parcel.q;
      const float ddq = fmaxf(zqsa - s_qe[k][lane], 0.f), ddt = ztp - s_te[k][lane];
      s_dq[k][lane] = ddq;
      s_dt[k][lane] = ddt;
      zpt = ddt * dsk * s_acpe[k][lane] + zpt;
      zpq = ddq * dsk * K.ALV + zpq;
      zbeta = fminf(1.f, s_qe[k][lane] / zqsa) * dsk + zbeta;
      zpbeta = zpbeta + dsk;
      zi = s_tot[k][lane] * dsk * K.ALV + zi;
    }
    zi = fmaxf(0.f, zi);
    const float zrhm = zpbeta > 0.f ? zbeta / zpbeta : 0.f;
    float beta = 1.f;
    if (zrhm >= K.RHBETA) beta = powi((1.f - zrhm) / (1.f - K.RHBETA), (int)K.NBETA);
    s_zi[lane] = zi;
    s_zat[lane] = zpt > 0.f ? zi * (1.f - beta) / zpt : 0.f;
    s_zaq[lane] = zpq > 0.f ? zi * beta / zpq : 0.f;
    s_ilift[lane] = ilift;
    s_itop[lane] = itop;
  }
  __syncthreads();
  const int ilift = s_ilift[lane], itop = s_itop[lane];
  const float zi = s_zi[lane];
  const bool shallow = itop > 0 && (dp * sg[itop - 1] > K.PDEEP || zi <= 0.f);
  {
    const int level = l + 1;
    const float zat = s_zat[lane], zaq = s_zaq[lane];
    float dprcl = 0.f, icclev = 0.f;
    if (ilift >= level && itop <= level && zi > 0.f && !shallow) {
      const float zalcpe = K.ALV / zacpe;
      F.dqdt[at] = zaq * s_dq[l][lane] / D2 - zdqt;
      F.dtdt[at] = zat * s_dt[l][lane] / D2 + dtdt_in;
      dprcl = zat * s_dt[l][lane] * dsl / zalcpe / D2;
    }
    if (dprcl > 0.f) icclev = 1.f;
    s_flag[l][lane] = dprcl > 0.f;
    if (sgl < 0.4f && icclev == 1.f && itop == level) icclev = 2.f;
    F.dprcl[at] = dprcl;
    F.dprscl[at] = 0.f;
    F.icclev[at] = icclev;
  }
  if (!__syncthreads_or(shallow)) {
    if (l == 0) {
      float icctot = 0.f;
      for (int k = 0; k < NL; ++k) icctot = icctot + (float)s_flag[k][lane];
      F.icctot[c] = icctot;
    }
    return;
  }
  if (l == 0) {
    float icctot = 0.f;
    for (int k = 0; k < NL; ++k) icctot = icctot + (float)s_flag[k][lane];
    F.icctot[c] = icctot;
  }
  // mkshallow, for the block if any of its columns is shallow
  const float zkonst1 = K.GA * D2 / K.GASCON;
  const float zkonst2 = K.RKSHALLOW * zkonst1 * K.GA / K.GASCON;
  float zkdiff = 0.f;
  if (l < NM) {
    int kktop = 1;
    for (int level = 2; level <= NM; ++level)
      if (dp * sg[level - 1] < K.PDEEPTH) kktop = level;
    const int ktop = max(itop, kktop);
    const int lp = l + 1, level = l + 1;
    const float ztep = s_te[lp][lane];
    const float sigmah = tb[m.to.sigmah + l];
    const float zfac = zkonst2 * sigmah * sigmah * tb[m.to.vdiff_rdsig + l];
    const float dsp = ds[lp];
    const float zrthl = (dsp + dsl) / sum_products(zte, dsp, ztep, dsl);
    if (level >= ktop && level < ilift) zkdiff = zfac * zrthl * zrthl;
    if (level + 1 == ktop) {
      float zzqs = sat_capped(K, zte, dp * sgl);
      zzqs = zzqs * (1.f / (1.f - K.MOIST * zzqs));
      float zzqsp = sat_capped(K, ztep, dp * sg[lp]);
      zzqsp = zzqsp * (1.f / (1.f - K.MOIST * zzqsp));
      const float zrh = zqe / zzqs, zrhp = s_qe[lp][lane] / zzqsp;
      const float zzf = fabsf((zrh - 0.8f) / 0.2f * (zrhp - zrh));
      zkdiff = zfac * zrthl * zrthl * zzf;
    }
  }
  s_kq[l][lane] = zkdiff;
  s_kt[l][lane] = l < NM ? zkdiff * tb[m.to.vdiff_skaph + l] : zkdiff;
  __syncthreads();
  if (l == 0 && shallow)
    diffuse_column<NL, kCols>(ds, &s_qe[0][lane], &s_kq[0][lane], &s_pt[0][lane]);
  else if (l == 1 && shallow)
    diffuse_potential_column<NL, kCols>(ds, &s_te[0][lane], &s_kt[0][lane], tb + m.to.vdiff_skap, &s_pq[0][lane]);
  __syncthreads();
  if (!shallow) return;
  F.dtdt[at] = dtdt_in + (s_te[l][lane] - zte) / D2;
  F.dqdt[at] = dqdt_in + (s_qe[l][lane] - zqe) / D2;
}

#define LEVEL_LAUNCHER(name, kernel)                                                                          \
  template <int NL>                                                                                           \
  struct name {                                                                                               \
    static void run(const Model& m, cudaStream_t st) {                                                        \
      step_launch(m.column_pdl, kernel<NL>, (unsigned)((size_t)m.d.S * m.d.NHOR / kCols), 32 * NL, 0, st, m, m.pc, \
                  m.tabs);                                                                                    \
    }                                                                                                         \
  };
LEVEL_LAUNCHER(RainLevels, k_rain_levels)
LEVEL_LAUNCHER(KuoLevels, k_kuo_levels)

}  // namespace

// us a launch, a thread per column against a thread per (column, level), at
// columns x levels (CUDA events): rain 2,048 x 10 14.3 / 7.0, 8,192 x 10 14.6 /
// 8.2, 18,432 x 10 16.5 / 14.5, 24,576 x 10 16.5 / 16.5, 32,768 x 10 16.5 / 22.2;
// kuo 7.4 / 3.7, 7.4 / 4.0, 14.5 / 8.5, 10.4 / 10.4, 10.4 / 13.8. The line is ten
// levels'. With five, whose blocks have half the warps, the second form still
// wins somewhat above it: a step of T21 L5 planets 95 / 88 at 2,048 columns, 144 /
// 136 at 20,480, 144 / 131 at 24,576, 154 / 141 at 32,768, 166 / 176 at 49,152.
bool phy_levels(const Model& m) { return (long)m.d.S * m.d.NHOR <= 20480; }

void lev_rain(const Model& m, cudaStream_t st) { by_levels<RainLevels>(m.d.L, m, st); }
void lev_kuo(const Model& m, cudaStream_t st) { by_levels<KuoLevels>(m.d.L, m, st); }

}  // namespace exogcm
