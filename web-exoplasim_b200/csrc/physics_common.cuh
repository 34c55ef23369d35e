// Shared helpers of the column-physics translation units (physics.cu and
// physics_flux.cu): the column prologues, saturation and power helpers, the
// per-level-count dispatch and the one-thread-per-column launcher.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <string>

#include "common.cuh"
#include "launch.h"

namespace exogcm {

namespace {

constexpr int kBlock = 128;

// Asks L2 for a line this thread reads after its first store, so that load
// then hits L2 instead of DRAM (a hint: it moves no data into registers).
__device__ __forceinline__ void prefetch_l2(const float* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Column kernels take the planet constants and per-planet tables as
// __restrict__ parameters: both are read-only during a launch, so the
// compiler may keep their values across the kernel's stores to fields
// instead of reloading them after every store.
#define COLUMN_PROLOGUE                                              \
  pdl_wait();                                                        \
  pdl_release();                                                     \
  const Dims& d = m.d;                                               \
  const int c = blockIdx.x * blockDim.x + threadIdx.x;               \
  if (c >= d.S * d.NHOR) return;                                     \
  const int slot = c / d.NHOR;                                       \
  const int h = c % d.NHOR;                                          \
  const StepParams& P = m.params[slot];                              \
  if (!P.active) return;                                             \
  const PlanetConst& K = pcr[slot];                                  \
  const float* tb = tabr + (size_t)slot * m.to.stride;               \
  const size_t SN = (size_t)d.S * d.NHOR;                            \
  const FieldPtrs& F = m.f;                                          \
  (void)h; (void)K; (void)tb; (void)SN; (void)F; (void)P;

// The same for a kernel that reads its planet's constants inside long
// loops: column kernels run kBlock threads per block over S * NHOR columns,
// and kBlock divides NHOR (2048, 8192 or 18432), so a block's columns
// belong to one slot, whose constants are staged once in shared memory.
#define COLUMN_PROLOGUE_STAGED                                       \
  pdl_wait();                                                        \
  pdl_release();                                                     \
  const Dims& d = m.d;                                               \
  const int slot = blockIdx.x * kBlock / d.NHOR;                     \
  const StepParams& P = m.params[slot];                              \
  if (!P.active) return;                                             \
  __shared__ PlanetConst s_planet;                                   \
  stage_planet(pcr + slot, &s_planet);                               \
  const PlanetConst& K = s_planet;                                   \
  const int c = blockIdx.x * kBlock + threadIdx.x;                   \
  if (c >= d.S * d.NHOR) return;                                     \
  const int h = c - slot * d.NHOR;                                   \
  const float* tb = tabr + (size_t)slot * m.to.stride;               \
  const size_t SN = (size_t)d.S * d.NHOR;                            \
  const FieldPtrs& F = m.f;                                          \
  (void)h; (void)K; (void)tb; (void)SN; (void)F; (void)P;

// Copies one slot's constants into shared memory (all threads of the block
// take part and meet at the barrier).
__device__ __forceinline__ void stage_planet(const PlanetConst* src, PlanetConst* dst) {
  constexpr int n = sizeof(PlanetConst) / sizeof(float);
  const float* a = reinterpret_cast<const float*>(src);
  float* b = reinterpret_cast<float*>(dst);
  for (int i = threadIdx.x; i < n; i += blockDim.x) b[i] = a[i];
  __syncthreads();
}

__device__ __forceinline__ float sat_capped(const PlanetConst& K, float t, float p) {
  return fminf(K.RDBRV * K.RA1 * expf(K.RA2 * (t - K.TMELT) / (t - K.RA4)) / p, K.RDBRV);
}
// The same with IEEE divisions, for the large-scale condensation, whose
// precipitation is the small difference of two iterated states.
__device__ __forceinline__ float sat_capped_rn(const PlanetConst& K, float t, float p) {
  return fminf(__fdiv_rn(K.RDBRV * K.RA1 * expf(__fdiv_rn(K.RA2 * (t - K.TMELT), t - K.RA4)), p), K.RDBRV);
}
__device__ __forceinline__ float sat_divided(const PlanetConst& K, float t, float p) {
  const float q = sat_capped(K, t, p);
  return q / (1.f - K.MOIST * q);
}
// The longwave band fits' base-2 logarithm and power: CUDA's accurate
// log2f and exp2f, or, built with EXOGCM_LWR_FAST_LOG2 / EXOGCM_LWR_FAST_EXP2,
// the special-function unit's lg2.approx / ex2.approx instructions.
__device__ __forceinline__ float fit_log2(float x) {
#ifdef EXOGCM_LWR_FAST_LOG2
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return log2f(x);
#endif
}
__device__ __forceinline__ float fit_exp2(float x) {
#ifdef EXOGCM_LWR_FAST_EXP2
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return exp2f(x);
#endif
}
// x^y for x >= 0 with 0^y = 0: precise_pow (src/model/shared/gpu/math/wgsl/
// precise.wgsl:100-103) is exp(y * log(x)); here exp2(y * log2(x)) with
// CUDA's own exp2f and log2f.
__device__ __forceinline__ float fpow(float x, float y) {
#ifdef EXOGCM_FAST_POW
  float l, r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y * l));
  return x == 0.f ? 0.f : r;
#else
  return x == 0.f ? 0.f : exp2f(y * log2f(x));
#endif
}
// x^n by binary exponentiation, as libgcc's __powisf2 computes x**n.
__device__ __forceinline__ float powi(float x, int n) {
  float base = x;
  unsigned mm = (unsigned)abs(n);
  float result = (mm & 1u) ? x : 1.f;
  mm >>= 1;
  while (mm) {
    base = base * base;
    if (mm & 1u) result = result * base;
    mm >>= 1;
  }
  return n < 0 ? 1.f / result : result;
}

constexpr float kPI = 3.14159265359f;
constexpr float kTWOPI = kPI + kPI;

constexpr int kSumThreads = 256;

inline unsigned nblocks(size_t n, int b) { return (unsigned)((n + b - 1) / b); }

// Implicit vertical diffusion (physics/diffusion/wgsl/implicit.wgsl): the
// tridiagonal solve of one column, for a quantity and for potential
// temperature, with IEEE divisions (the tendencies are small differences of
// the diffused and the old profiles). Exchange coefficients and humidities
// are often zero, hence quotient: vdiff 203 -> 193 us and kuo (mkshallow) 119
// -> 112 at 128 T42 L10 planets, kuo 12.5 -> 7.6 at one T21 L10 planet.
template <int NL>
__device__ __forceinline__ void diffuse(const float* ds, float* x, const float* k) {
  float ebs[NL];
  const float ds0 = ds[0];
  ebs[0] = quotient(k[0], ds0 + k[0]);
  x[0] = quotient(ds0 * x[0], ds0 + k[0]);
#pragma unroll
  for (int l = 1; l < NL - 1; ++l) {
    const float den = ds[l] + k[l] + k[l - 1] * (1.f - ebs[l - 1]);
    ebs[l] = quotient(k[l], den);
    x[l] = quotient(x[l] * ds[l] + k[l - 1] * x[l - 1], den);
  }
  const float dsn = ds[NL - 1];
  x[NL - 1] = quotient(x[NL - 1] * dsn + k[NL - 2] * x[NL - 2], dsn + k[NL - 2] * (1.f - ebs[NL - 2]));
#pragma unroll
  for (int l = NL - 2; l >= 0; --l) x[l] = x[l] + ebs[l] * x[l + 1];
}

template <int NL>
__device__ __forceinline__ void diffuse_potential(const float* ds, float* x, const float* k, const float* skap) {
  float ebs[NL];
  const float ds0 = ds[0];
  ebs[0] = quotient(k[0], ds0 + quotient(k[0], skap[0]));
  x[0] = quotient(ds0 * x[0], ds0 + quotient(k[0], skap[0]));
#pragma unroll
  for (int l = 1; l < NL - 1; ++l) {
    const float den = ds[l] + quotient(k[l] + k[l - 1] * (1.f - quotient(ebs[l - 1], skap[l - 1])), skap[l]);
    ebs[l] = quotient(k[l], den);
    x[l] = quotient(x[l] * ds[l] + quotient(k[l - 1], skap[l - 1]) * x[l - 1], den);
  }
  const int last = NL - 1;
  const float dsn = ds[last];
  x[last] = quotient(x[last] * dsn + quotient(k[NL - 2] * x[NL - 2], skap[NL - 2]),
                      dsn + quotient(k[NL - 2], skap[last]) * (1.f - quotient(ebs[NL - 2], skap[NL - 2])));
#pragma unroll
  for (int l = NL - 2; l >= 0; --l) x[l] = x[l] + quotient(ebs[l] * x[l + 1], skap[l + 1]);
}


// a b + c d with the first product fused, as the compiler forms the sums of
// diffuse and k_kuo that have two products to choose from.
__device__ __forceinline__ float sum_products(float a, float b, float c, float d) {
  return __fmaf_rn(a, b, __fmul_rn(c, d));
}

// The implicit vertical diffusion of one column in shared memory (diffuse,
// diffuse_potential above): the same solves, the level loop rolled. x and k
// are the column's levels, STRIDE apart; ebs is scratch.
template <int NL, int STRIDE>
__device__ __forceinline__ void diffuse_column(const float* __restrict__ ds, float* x, const float* k, float* ebs) {
  const float ds0 = ds[0], k0 = k[0];
  float e = quotient(k0, ds0 + k0), v = quotient(ds0 * x[0], ds0 + k0), kp = k0;
  ebs[0] = e;
  x[0] = v;
#pragma unroll 1
  for (int l = 1; l < NL - 1; ++l) {
    const float kl = k[l * STRIDE];
    const float den = ds[l] + kl + kp * (1.f - e);
    e = quotient(kl, den);
    v = quotient(sum_products(x[l * STRIDE], ds[l], kp, v), den);
    ebs[l * STRIDE] = e;
    x[l * STRIDE] = v;
    kp = kl;
  }
  const float dsn = ds[NL - 1];
  v = quotient(sum_products(x[(NL - 1) * STRIDE], dsn, kp, v), dsn + kp * (1.f - e));
  x[(NL - 1) * STRIDE] = v;
#pragma unroll 1
  for (int l = NL - 2; l >= 0; --l) {
    v = x[l * STRIDE] + ebs[l * STRIDE] * v;
    x[l * STRIDE] = v;
  }
}

template <int NL, int STRIDE>
__device__ __forceinline__ void diffuse_potential_column(const float* __restrict__ ds, float* x, const float* k,
                                                         const float* __restrict__ skap, float* ebs) {
  const float ds0 = ds[0], k0 = k[0];
  float e = quotient(k0, ds0 + quotient(k0, skap[0]));
  float v = quotient(ds0 * x[0], ds0 + quotient(k0, skap[0]));
  float kp = k0;
  ebs[0] = e;
  x[0] = v;
#pragma unroll 1
  for (int l = 1; l < NL - 1; ++l) {
    const float kl = k[l * STRIDE], sp = skap[l - 1];
    const float den = ds[l] + quotient(kl + kp * (1.f - quotient(e, sp)), skap[l]);
    e = quotient(kl, den);
    v = quotient(sum_products(x[l * STRIDE], ds[l], quotient(kp, sp), v), den);
    ebs[l * STRIDE] = e;
    x[l * STRIDE] = v;
    kp = kl;
  }
  const int last = NL - 1;
  const float dsn = ds[last], sp = skap[NL - 2];
  v = quotient(x[last * STRIDE] * dsn + quotient(kp * v, sp), dsn + quotient(kp, skap[last]) * (1.f - quotient(e, sp)));
  x[last * STRIDE] = v;
#pragma unroll 1
  for (int l = NL - 2; l >= 0; --l) {
    v = x[l * STRIDE] + quotient(ebs[l * STRIDE] * v, skap[l + 1]);
    x[l * STRIDE] = v;
  }
}

// Clear-sky longwave transmissivity for absorber sums (lwr.wgsl's band fits).
// Each fit is a power law below its threshold and a logarithm above; both
// sides are written through one base-2 logarithm of the side's argument,
// x^y = 2^(y log2 x) and log10 x = log10(2) log2 x, so that the columns of
// a warp, whichever side they take, share one instruction stream (no
// divergent branches) and two special-function operations per fit. All
// power-law arguments are positive.
__device__ __forceinline__ float lwr_clear_sky(const PlanetConst& K, float sumwv, float sumo3, float sumco2) {
  const float ZERO = 1.0e-6f, LOG10_2 = 0.30102999566398120f, LN_2 = 0.69314718055994531f;
  const bool wv1 = sumwv <= 0.01f, wv2 = sumwv <= 2.f, co2 = sumco2 <= 1.f, o3 = sumo3 <= 0.01f;
  const float lah = fit_log2(sumwv + (wv1 ? 3.59e-5f : 0.01f));
  const float lth = fit_log2(wv2 ? sumwv + 0.0286f : sumwv - 0.6931f);
  const float lco = fit_log2(co2 ? sumco2 + 0.01022f : sumco2);
  const float lo3 = fit_log2(o3 ? sumo3 + 7.0e-5f : sumo3);
  float ah2o = wv1 ? 0.846f * fit_exp2(0.243f * lah) - K.ZH2O0A : 0.24f * (LOG10_2 * lah) + K.ZAH2OC;
  if (K.TH2OC > 0.f) ah2o = fminf(ah2o + (1.f - expf(-K.TH2OC * sumwv)), 1.f);
  const float aco2 = co2 ? 0.0676f * fit_exp2(0.421f * lco) - K.ZCO20 : 0.0546f * (LOG10_2 * lco) + K.ZACO2C;
  const float th2o = wv2 ? 1.f - (0.832f * fit_exp2(0.26f * lth) - K.ZH2O0)
                         : fmaxf(0.f, K.ZTH2OC - 0.1196f * (LN_2 * lth));
  const float ao3 = o3 ? 0.209f * fit_exp2(0.436f * lo3) - K.ZAO30 : 0.0212f * (LOG10_2 * lo3) + K.ZAO3C;
  return fminf(1.f - ZERO, fmaxf(ZERO, 1.f - ah2o - ao3 - aco2 * th2o));
}

struct Parcel {
  float t, q, cor;
  bool saturated;
};

// kuo.wgsl's condense: a lifted parcel's two Newton condensation steps.
__device__ __forceinline__ Parcel condense(const PlanetConst& K, float t0, float q0, float p) {
  float s = sat_capped(K, t0, p);
  float cor = 1.f / (1.f - K.MOIST * s);
  s = s * cor;
  if (!(s < q0)) return {t0, q0, cor, false};
  float t = t0, q = q0;
  const float lcp = (t0 < K.TMELT ? K.ALS : K.ALV) / (K.ACPD * (1.f + K.ADV * q0));
  for (int i = 0; i < 2; ++i) {
    if (i == 1) {
      s = sat_capped(K, t, p);
      cor = 1.f / (1.f - K.MOIST * s);
      s = s * cor;
    }
    const float dqsdt = K.RA2 * (K.TMELT - K.RA4) * s * cor / ((t - K.RA4) * (t - K.RA4));
    const float rain = (q - s) / (1.f + lcp * dqsdt);
    t = t + lcp * rain;
    q = q - rain;
  }
  return {t, q, cor, true};
}

// |(u, v)| with both squares rounded before the sum (no contraction), the
// same wherever the speed is formed.
__device__ __forceinline__ float wind_speed(float u, float v) {
  return sqrtf(__fadd_rn(__fmul_rn(u, u), __fmul_rn(v, v)));
}

template <template <int> class Launch, typename... A>
void by_levels(int L, A&&... a) {
  if (L == 10)
    Launch<10>::run(a...);
  else if (L == 5)
    Launch<5>::run(a...);
}

// Column kernels begin with COLUMN_PROLOGUE(_STAGED), whose pdl_wait comes
// before any state access, so they start by programmatic dependent launch.
#define COLUMN_LAUNCHER(name, kernel)                                                               \
  template <int NL>                                                                                 \
  struct name {                                                                                     \
    static void run(const Model& m, cudaStream_t st) {                                              \
      step_launch(m.column_pdl, kernel<NL>, nblocks((size_t)m.d.S * m.d.NHOR, kBlock), kBlock, 0, st, m, m.pc, m.tabs); \
    }                                                                                               \
  };

}  // namespace

}  // namespace exogcm
