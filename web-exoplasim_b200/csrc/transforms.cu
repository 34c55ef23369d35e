// Longitude (Fourier) and latitude (Gauss-Legendre) transforms, batched over
// every plane of every planet slot, in plain FP32 on the CUDA cores.
//
// Semantics follow the reference's WGSL transforms
// (src/model/climate/gcm/fourier/wgsl/*.wgsl, legendre/wgsl/*.wgsl): the
// longitude transforms are the truncated DFT with the f64-built tables of
// fourier/index.ts:19-36 (c_m = (1/N) sum_j g_j e^{-i m lambda_j} for
// m <= NTRU, and its inverse that ignores Im c_0), and the Legendre sums run
// over latitude pairs with the (m + n)-parity folding of legmod's
// single-process branch. Each kernel stages what its threads share in shared
// memory: the DFT tables and a tile of rows, or a tile of spectral or Fourier
// planes, so each table element read from L2 serves a whole tile.
#include <cuda_runtime.h>

#include <algorithm>

#include "async_copy.cuh"
#include "common.cuh"
#include "launch.h"

namespace exogcm {

namespace {

// ---------------------------------------------------------------- DFTs
// gp2fc and fc2gp of the plain path as one dense product: row r of `in` (K
// values) times the table [K][N], N columns out, summed over K in order as
// the shaders do. A block stages the table once and walks chunks of R rows;
// a thread owns two adjacent columns of four rows, so a table pair and a
// row's four K values loaded from shared memory serve 8 and 2 multiply-adds.
// What bounds it is the shared-memory loads (12 wavefronts per 32 warp-wide
// multiply-adds). One thread per output with the table staged by each of 20
// blocks took 39 us for one T42 L10 planet's field, whatever its number of
// rows: a chain of 128 loads and multiply-adds behind a 44 KB staging on 20
// SMs. A launch now takes every field of a stage.
constexpr int kDftRows = 4;  // rows per thread

__global__ void __launch_bounds__(768) k_dft(const __grid_constant__ TrSet set, const float* __restrict__ tab, int K,
                                             int N, int nlat, int R, int items) {
  extern __shared__ float4 dft_smem[];
  const int KP = (K + 3) / 4 * 4;  // row pitch: rows start 16-byte aligned
  float* ts = reinterpret_cast<float*>(dft_smem);  // [K][N]
  float* rs = ts + (K * N + 3) / 4 * 4;            // [R][KP]
  for (int i = threadIdx.x; i < K * N / 4; i += blockDim.x) cp_async16(ts + 4 * i, tab + 4 * i);
  pdl_wait();
  pdl_release();
  const int pairs = N / 2, chunks = nlat / R;
  const int col = 2 * (threadIdx.x % pairs), r0 = kDftRows * (threadIdx.x / pairs);
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int tile = item / chunks, fi = tr_find(set, tile);
    const size_t row0 = (size_t)(tile - set.at[fi]) * nlat + (item % chunks) * R;
    const float* in = set.f[fi].a + row0 * K;
    for (int i = threadIdx.x; i < R * (K / 2); i += blockDim.x) {
      const int r = i / (K / 2), k = 2 * (i - r * (K / 2));
      cp_async8(rs + r * KP + k, in + (size_t)r * K + k);
    }
    cp_async_wait_all();
    __syncthreads();
    const int ncol = set.f[fi].opt ? 2 * set.f[fi].opt : N;  // gp2fc: wavenumbers written
    if (r0 < R && col < ncol) {
      float2 s[kDftRows] = {};
      const float* tc = ts + col;
      const float* rr = rs + r0 * KP;
      auto add = [&](int k, float x0, float x1, float x2, float x3) {
        const float2 t = *reinterpret_cast<const float2*>(tc + k * N);
        s[0] = make_float2(fmaf(t.x, x0, s[0].x), fmaf(t.y, x0, s[0].y));
        s[1] = make_float2(fmaf(t.x, x1, s[1].x), fmaf(t.y, x1, s[1].y));
        s[2] = make_float2(fmaf(t.x, x2, s[2].x), fmaf(t.y, x2, s[2].y));
        s[3] = make_float2(fmaf(t.x, x3, s[3].x), fmaf(t.y, x3, s[3].y));
      };
      int k = 0;
#pragma unroll 2
      for (; k + 3 < K; k += 4) {
        float4 x[kDftRows];
#pragma unroll
        for (int i = 0; i < kDftRows; ++i) x[i] = *reinterpret_cast<const float4*>(rr + i * KP + k);
        add(k, x[0].x, x[1].x, x[2].x, x[3].x);
        add(k + 1, x[0].y, x[1].y, x[2].y, x[3].y);
        add(k + 2, x[0].z, x[1].z, x[2].z, x[3].z);
        add(k + 3, x[0].w, x[1].w, x[2].w, x[3].w);
      }
      for (; k < K; ++k) add(k, rr[k], rr[KP + k], rr[2 * KP + k], rr[3 * KP + k]);
      float* out = set.f[fi].x + (row0 + r0) * N + col;
#pragma unroll
      for (int i = 0; i < kDftRows; ++i) *reinterpret_cast<float2*>(out + (size_t)i * N) = s[i];
    }
    __syncthreads();  // the next chunk restages the rows
  }
}

// gpmt: d/dlambda in Fourier space, (re, im) * i m (fourier/wgsl/dlambda.wgsl).
__global__ void k_dlambda(const float* a, float* b, int n, int ntp1, int nfc) {
  pdl_wait();
  pdl_release();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int m = i % ntp1;
  const size_t at = (size_t)(i / ntp1) * nfc + 2 * m;
  const float re = a[at], im = a[at + 1];
  b[at] = -im * (float)m;
  b[at + 1] = re * (float)m;
}

// The same on the optimized path's m-major Fourier planes (coefficient
// (m, lat) at 2 * (m * NLAT + lat)).
__global__ void k_dlambda_m_major(const float* a, float* b, int n, int nlat, int ntp1) {
  pdl_wait();
  pdl_release();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int m = (i / nlat) % ntp1;
  const size_t at = 2 * (size_t)i;
  const float re = a[at], im = a[at + 1];
  b[at] = -im * (float)m;
  b[at + 1] = re * (float)m;
}

// ---------------------------------------------------------------- Legendre
// Inverse transforms (sp2fc, sp2fcdmu, dv2uv): output (plane, lat, m) sums
// modes n = m..NTRU of its plane. A block stages a tile of spectral planes
// and the table rows of a tile of latitudes in shared memory, and each
// thread computes wavenumbers j and NTRU - j of one (plane, latitude)
// together, so every thread sums NTRU + 2 terms. The tiles are small (two
// planes by four or eight latitudes) because the path steps single planets:
// four planes by sixteen latitudes left one planet's field 12 blocks (49 us
// at T42 L10), and a launch takes every field of a stage.
constexpr int kInvPlanes = 2;
constexpr int kInvLats = 8, kDvLats = 4;  // latitudes per block: sp2fc, dv2uv (divide every NLAT)

__device__ __forceinline__ int mode_first(int m, int ntp1) { return m * (2 * ntp1 - m + 1) / 2; }

// Copies `n` floats (both 8-byte aligned, n even).
__device__ __forceinline__ void copy_floats(float* dst, const float* src, int n) {
  for (int i = threadIdx.x; i < n / 2; i += blockDim.x) cp_async8(dst + 2 * i, src + 2 * i);
}

__global__ void k_leg_inverse(const __grid_constant__ TrSet set, const float* __restrict__ qi,
                              const float* __restrict__ qj, Dims d) {
  extern __shared__ float4 inv_smem[];
  float* sp = reinterpret_cast<float*>(inv_smem);  // [kInvPlanes][NRSP]
  float* qs = sp + kInvPlanes * d.NRSP;            // [kInvLats][NCSP]
  const int fi = tr_find(set, blockIdx.x);
  const int p0 = (blockIdx.x - set.at[fi]) * kInvPlanes;
  const int np = min(kInvPlanes, set.f[fi].planes - p0);
  const int lat0 = blockIdx.y * kInvLats;
  const float* q = set.f[fi].opt & kTrDerivative ? qj : qi;
  copy_floats(qs, q + (size_t)lat0 * d.NCSP, kInvLats * d.NCSP);
  pdl_wait();
  pdl_release();
  copy_floats(sp, set.f[fi].a + (size_t)p0 * d.NRSP, np * d.NRSP);
  cp_async_wait_all();
  __syncthreads();
  const int pairs = (d.NTP1 + 1) / 2;
  for (int o = threadIdx.x; o < np * kInvLats * pairs; o += blockDim.x) {
    const int j = o % pairs;
    const int lat = (o / pairs) % kInvLats;
    const int p = o / (pairs * kInvLats);
    const float* spp = sp + p * d.NRSP;
    const float* qr = qs + lat * d.NCSP;
    float* out = set.f[fi].x + ((size_t)(p0 + p) * d.NLAT + lat0 + lat) * d.NFC;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const int m = half == 0 ? j : d.T - j;
      if (half == 1 && m == j) break;
      const int first = mode_first(m, d.NTP1);
      float re = 0.f, im = 0.f;
#pragma unroll 4
      for (int w = first; w < first + d.NTP1 - m; ++w) {
        const float qq = qr[w];
        const float2 v = *reinterpret_cast<const float2*>(spp + 2 * w);
        re = fmaf(qq, v.x, re);
        im = fmaf(qq, v.y, im);
      }
      *reinterpret_cast<float2*>(out + 2 * m) = make_float2(re, im);
    }
  }
}

// dv2uv: winds at every latitude from spectral divergence and vorticity,
// with plavor removed from vorticity mode w = 1 (legendre/wgsl/dv2uv.wgsl).
__global__ void k_dv2uv(const __grid_constant__ TrSet set, const float* __restrict__ qu,
                        const float* __restrict__ qv, Dims d) {
  extern __shared__ float4 inv_smem[];
  float* dd0 = reinterpret_cast<float*>(inv_smem);    // [kInvPlanes][NRSP]
  float* zz0 = dd0 + kInvPlanes * d.NRSP;             // [kInvPlanes][NRSP]
  float* qus = zz0 + kInvPlanes * d.NRSP;             // [kDvLats][NCSP]
  float* qvs = qus + kDvLats * d.NCSP;                // [kDvLats][NCSP]
  const int fi = tr_find(set, blockIdx.x);
  const int p0 = (blockIdx.x - set.at[fi]) * kInvPlanes;
  const int np = min(kInvPlanes, set.f[fi].planes - p0);
  const int lat0 = blockIdx.y * kDvLats;
  copy_floats(qus, qu + (size_t)lat0 * d.NCSP, kDvLats * d.NCSP);
  copy_floats(qvs, qv + (size_t)lat0 * d.NCSP, kDvLats * d.NCSP);
  pdl_wait();
  pdl_release();
  copy_floats(dd0, set.f[fi].a + (size_t)p0 * d.NRSP, np * d.NRSP);
  copy_floats(zz0, set.f[fi].b + (size_t)p0 * d.NRSP, np * d.NRSP);
  cp_async_wait_all();
  __syncthreads();
  if (threadIdx.x < np) zz0[threadIdx.x * d.NRSP + 2] -= set.f[fi].plavor;  // w == 1, real part
  __syncthreads();
  const int pairs = (d.NTP1 + 1) / 2;
  for (int o = threadIdx.x; o < np * kDvLats * pairs; o += blockDim.x) {
    const int j = o % pairs;
    const int lat = (o / pairs) % kDvLats;
    const int p = o / (pairs * kDvLats);
    const float* dd = dd0 + p * d.NRSP;
    const float* zz = zz0 + p * d.NRSP;
    const float* qur = qus + lat * d.NCSP;
    const float* qvr = qvs + lat * d.NCSP;
    const size_t row = ((size_t)(p0 + p) * d.NLAT + lat0 + lat) * d.NFC;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const int m = half == 0 ? j : d.T - j;
      if (half == 1 && m == j) break;
      const int first = mode_first(m, d.NTP1);
      float ure = 0.f, uim = 0.f, vre = 0.f, vim = 0.f;
#pragma unroll 4
      for (int w = first; w < first + d.NTP1 - m; ++w) {
        const float a = qur[w], b = qvr[w];
        const float zre = zz[2 * w], zim = zz[2 * w + 1], dre = dd[2 * w], dim = dd[2 * w + 1];
        ure = ure + b * zre + a * dim;
        uim = uim + b * zim - a * dre;
        vre = vre + a * zim - b * dre;
        vim = vim - a * zre - b * dim;
      }
      *reinterpret_cast<float2*>(set.f[fi].x + row + 2 * m) = make_float2(ure, uim);
      *reinterpret_cast<float2*>(set.f[fi].y + row + 2 * m) = make_float2(vre, vim);
    }
  }
}

// Dynamic shared memory above 48 KB needs an opt-in per kernel; tr_init sets
// it once for every transform kernel before any launch or graph capture.
constexpr int kMaxDynamicSmem = 200 * 1024;
template <typename K>
void allow_smem(K kernel) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
}

// Rows per DFT chunk (dividing every NLAT): the most that still gives every
// SM a chunk, so that one planet's few rows spread over the chip and a
// batch's many rows reuse a staged table pair 8 times.
int dft_rows(const Dims& d, int planes) {
  for (int r : {32, 16})
    if (planes * (d.NLAT / r) >= sm_count()) return r;
  return 8;
}

void launch_dft(const Model& m, TrSet set, const float* tab, int K, int N, cudaStream_t st) {
  const int planes = tr_tiles(set, 1);
  const int R = dft_rows(m.d, planes);
  const int items = planes * (m.d.NLAT / R);
  const size_t smem = ((size_t)(K * N + 3) / 4 * 4 + (size_t)R * ((K + 3) / 4 * 4)) * sizeof(float);
  const int threads = N / 2 * (R / kDftRows);
  const int grid = std::min(items, persistent_grid((const void*)k_dft, threads, smem));
  step_launch(m.pdl, k_dft, grid, threads, smem, st, set, tab, K, N, m.d.NLAT, R, items);
}

}  // namespace

void tr_init() {
  leg_init();
  tc_init();
  fft_init();
  grid_init();
  allow_smem(k_dft);
  allow_smem(k_leg_inverse);
  allow_smem(k_dv2uv);
}

void tr_fourier_forward(const Model& m, TrSet s, cudaStream_t st) {
  if (m.mode >= 1) return fft_forward(m, s, st);
  launch_dft(m, s, m.sh.fwd, m.d.NLON, m.d.NFC, st);
}

void tr_fourier_inverse(const Model& m, TrSet s, cudaStream_t st) {
  if (m.mode >= 1) return fft_inverse(m, s, st);
  launch_dft(m, s, m.sh.inv, m.d.NFC, m.d.NLON, st);
}

static void dlambda(const Model& m, const float* a, float* b, int planes, cudaStream_t st) {
  const int n = planes * m.d.NLAT * m.d.NTP1;
  const unsigned grid = (n + 255) / 256;
  if (m.mode >= 1)
    step_launch(m.pdl, k_dlambda_m_major, grid, 256, 0, st, a, b, n, m.d.NLAT, m.d.NTP1);
  else
    step_launch(m.pdl, k_dlambda, grid, 256, 0, st, a, b, n, m.d.NTP1, m.d.NFC);
}

void tr_spectral_part(const Model& m, const TrSet& s, cudaStream_t st) {
  if (m.mode == 1) return grid_sp2gp(m, s, st);
  // sp2fc of every field that is not another's d/dlambda, then d/dlambda
  // from the field sharing its spectral input
  TrSet inv;
  for (int i = 0; i < s.n; ++i)
    if (!(s.f[i].opt & kTrDlambda)) inv.add(s.f[i]);
  tr_legendre_inverse(m, inv, st);
  for (int i = 0; i < s.n; ++i) {
    if (!(s.f[i].opt & kTrDlambda)) continue;
    const float* from = nullptr;
    for (int k = 0; k < s.n; ++k)
      if (s.f[k].a == s.f[i].a && !(s.f[k].opt & (kTrDlambda | kTrDerivative))) from = s.f[k].x;
    if (!from) throw std::logic_error("transform launch: d/dlambda of a field not in the set");
    dlambda(m, from, s.f[i].x, s.f[i].planes, st);
  }
}

void tr_grid_part(const Model& m, const TrSet& s, TrSet fourier, cudaStream_t st) {
  if (m.mode != 1)
    for (int i = 0; i < s.n; ++i) {
      TrField t;
      t.a = s.f[i].x;
      t.x = s.f[i].y;
      t.planes = s.f[i].planes;
      fourier.add(t);
    }
  if (fourier.n) tr_fourier_inverse(m, fourier, st);
}

void tr_legendre_inverse(const Model& m, TrSet s, cudaStream_t st) {
  if (m.mode == 2) return tc_inverse(m, s, st);
  if (m.mode == 1) return leg_inverse(m, s, st);
  const dim3 grid(tr_tiles(s, kInvPlanes), m.d.NLAT / kInvLats);
  const int threads = (kInvPlanes * kInvLats * ((m.d.NTP1 + 1) / 2) + 31) / 32 * 32;
  const size_t smem = ((size_t)kInvPlanes * m.d.NRSP + (size_t)kInvLats * m.d.NCSP) * sizeof(float);
  step_launch(m.pdl, k_leg_inverse, grid, threads, smem, st, s, m.sh.qi, m.sh.qj, m.d);
}

void tr_dv2uv(const Model& m, TrSet s, cudaStream_t st) {
  if (m.mode == 2) return tc_dv2uv(m, s, st);
  if (m.mode == 1) return leg_dv2uv(m, s, st);
  const dim3 grid(tr_tiles(s, kInvPlanes), m.d.NLAT / kDvLats);
  const int threads = (kInvPlanes * kDvLats * ((m.d.NTP1 + 1) / 2) + 31) / 32 * 32;
  const size_t smem = ((size_t)2 * kInvPlanes * m.d.NRSP + (size_t)2 * kDvLats * m.d.NCSP) * sizeof(float);
  step_launch(m.pdl, k_dv2uv, grid, threads, smem, st, s, m.sh.qu, m.sh.qv, m.d);
}

// The latitude-pair kernels sum in the shaders' order, so the plain path's
// forward transforms run on them too (on its own Fourier layout).
void tr_legendre_forward(const Model& m, TrSet s, cudaStream_t st) {
  m.mode == 2 ? tc_forward(m, s, st) : leg_forward(m, s, st);
}

void tr_uv2dv(const Model& m, TrSet s, cudaStream_t st) { m.mode == 2 ? tc_uv2dv(m, s, st) : leg_uv2dv(m, s, st); }

void tr_qtend(const Model& m, TrSet s, cudaStream_t st) { m.mode == 2 ? tc_qtend(m, s, st) : leg_qtend(m, s, st); }

}  // namespace exogcm
