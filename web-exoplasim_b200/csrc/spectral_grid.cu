// Inverse spectral transforms fused with the longitude FFT (optimized path):
// spectral plane -> grid plane in one kernel, so that the Fourier
// coefficients between sp2fc (legendre/wgsl/inverse.wgsl) and fc2gp
// (fourier/wgsl/inverse.wgsl) stay in shared memory instead of making a
// round trip through HBM.
//
// A block owns JR = 8 latitude pairs (16 rows of every plane) and walks a
// range of planes two (or four) at a time. Its slice of the northern table is
// copied in once (16-byte asynchronous copies of a slice laid out in HBM as
// it sits in shared memory), pair-major ([pair][mode]): a row pitch of 4
// (mod 32) banks and each
// wavenumber's modes starting at a position of residue m (mod 4) put the 32
// lanes of a warp (8 pairs x 4 consecutive wavenumbers) on 32 distinct banks.
// Per plane pair:
//  1. Legendre: lane (wavenumber m, latitude pair jj) sums the modes of m for
//     both planes: even-(n-m) and odd-(n-m) partial sums E, O in the order of
//     the unfused latitude-pair kernel (legendre.cu), north = E + O, south =
//     s (E - O). The Fourier coefficients go to the FFT's coefficient stage
//     [plane][m][row]. The warps take the groups of four wavenumbers, which
//     shorten with m, in snake order, so none sums much longer than another.
//     (Threads taking wavenumber pairs (u, NTP1 - 1 - u), all of one length,
//     did not divide evenly at T42: 704 pairs for 512 threads were two rounds,
//     the second a third full.)
//  2. FFT: the 32 rows of the pair, T threads per row, the four-step FFT of
//     fft.cu; rows are written to the grid plane.
// The next pair's spectral coefficients are fetched into registers during
// step 2, and the spectral stage shares its memory with the FFT's exchange
// rows. Results equal the unfused kernels' bit for bit. When the model asks
// to keep the Fourier fields (stage replay), or a field asks for it, step 1
// also writes them in the path's m-major layout.
//
// One launch takes the planes of several fields: passes of a block go from
// field to field (none spans two), the fields with the d/dmu table in blocks
// of their own. gp's d/dlambda is the coefficients times i m between the
// steps (fourier/wgsl/dlambda.wgsl). One launch for gridpointa's seven
// fields in place of nine kernels (sp2fc and d/dlambda, two FFTs, and a
// fused transform for each other field).
#include <cuda_runtime.h>

#include <algorithm>

#include "async_copy.cuh"
#include "common.cuh"
#include "fft_core.cuh"
#include "launch.h"

namespace exogcm {

// A block's slice of the northern table: JR latitude pairs, each a row of
// grid_table_pitch floats holding every mode, wavenumber m's modes from
// position grid_table_positions()[m]. The slices are laid out so in HBM
// once per resolution (grid_table_layout), and a block copies its slice
// into shared memory as it stands.
constexpr int kGridPairs = 8;

__host__ __device__ __forceinline__ int mode_start(int m, int ntp1) { return m * (2 * ntp1 - m + 1) / 2; }

// Row pitch: every mode plus up to 3 floats of alignment gap per wavenumber,
// rounded to 4 (mod 32) banks.
__host__ __device__ constexpr int grid_table_pitch(int ntp1) {
  return ntp1 * (ntp1 + 1) / 2 + 3 * ntp1 + ((((4 - (ntp1 * (ntp1 + 1) / 2 + 3 * ntp1)) % 32) + 32) % 32);
}

// m's modes start at a position of residue m (mod 4).
__host__ __device__ __forceinline__ void grid_table_positions(int ntp1, int* pos) {
  int at = 0;
  for (int m = 0; m < ntp1; ++m) {
    at += ((m - at) % 4 + 4) % 4;
    pos[m] = at;
    at += ntp1 - m;
  }
}

std::vector<float> grid_table_layout(const Dims& d, const std::vector<double>& qT) {
  const int JH = d.NLAT / 2, chunks = JH / kGridPairs, TP = grid_table_pitch(d.NTP1);
  std::vector<int> pos(d.NTP1);
  grid_table_positions(d.NTP1, pos.data());
  std::vector<float> out((size_t)chunks * kGridPairs * TP, 0.f);
  for (int c = 0; c < chunks; ++c)
    for (int jj = 0; jj < kGridPairs; ++jj) {
      float* row = out.data() + ((size_t)c * kGridPairs + jj) * TP;
      for (int m = 0, w = 0; m < d.NTP1; ++m)
        for (int k = 0; k < d.NTP1 - m; ++k, ++w) row[pos[m] + k] = (float)qT[(size_t)w * JH + c * kGridPairs + jj];
    }
  return out;
}

namespace {

using namespace fftcore;

template <int Q, int PPASS = 2>
struct GridShape {
  using F = Shape<Q>;
  static constexpr int M = F::M, N = F::N, NTP1 = F::NTP1, T = F::T;
  static constexpr int NLAT = M, JH = M / 2;
  static constexpr int NCSP = NTP1 * (NTP1 + 1) / 2;
  static constexpr int JR = kGridPairs;   // latitude pairs per block
  static constexpr int ROWS = 2 * JR;     // rows of a plane
  static constexpr int PP = PPASS;        // planes per pass (2 or 4)
  static constexpr int NPAIR = PP / 2;    // plane pairs per pass
  static constexpr int FROWS = PP * ROWS; // FFT rows per pass
  static constexpr int THREADS = FROWS * T;
  static constexpr int GROUPS = (NTP1 + 3) / 4;              // groups of four wavenumbers
  static constexpr int WARPS = THREADS / 32 / NPAIR;         // warps of a plane pair's Legendre sums
  static constexpr int TP = grid_table_pitch(NTP1);                // table row pitch, 4 (mod 32)
  static_assert((JR * TP) % 4 == 0, "a table slice is whole 16-byte chunks");
  static constexpr int PITCH = (ROWS + (((16 / T - ROWS) % 16) + 16) % 16);
  static constexpr int FC = NTP1 * PITCH;  // float2s of one plane's coefficient stage
  static constexpr int SPEC = NPAIR * NCSP;  // float4s of the spectral stage ([pair][mode], two planes each)
  static constexpr int XB = FROWS * 9 * Q;   // float2s of the FFT exchange rows
  static constexpr int SHARED = (2 * SPEC > XB ? 2 * SPEC : XB);  // float2s of the union
  static constexpr int R = (SPEC + THREADS - 1) / THREADS;        // spectral float4s per thread
  static_assert((N + 9 * Q + PP * FC) % 2 == 0, "the spectral stage must start 16-byte aligned");
  static_assert((N + 9 * Q + PP * FC + SHARED) % 2 == 0, "the table slice must start 16-byte aligned");
  static size_t smem() {
    return ((size_t)N + 9 * Q + (size_t)PP * FC + SHARED) * sizeof(float2) + (size_t)JR * TP * sizeof(float) +
           (size_t)NTP1 * sizeof(int);
  }
};

// Grid row of stage row rr of the block starting at pair j0: rows 0..JR-1
// are the northern latitudes j0.., rows JR..2JR-1 the southern ones in
// ascending order (NLAT - 2 JR - j0 + rr).
template <typename G>
__device__ __forceinline__ int stage_lat(int rr, int j0) {
  return rr < G::JR ? j0 + rr : G::NLAT - 2 * G::JR - j0 + rr;
}

// PP planes per pass: 2, or 4 (twice the threads and stages per block, the
// table slice and the barriers shared by twice the planes; the autotuner picks).
template <int Q, int PP>
__global__ void __launch_bounds__(GridShape<Q, PP>::THREADS)
    k_sp2gp(const __grid_constant__ TrSet set, int per_block, int passes0, int ranges0,
            const float* __restrict__ qi, const float* __restrict__ qj, const float2* __restrict__ twg, int keep_all) {
  using G = GridShape<Q, PP>;
  constexpr int T = G::T, M = G::M, N = G::N, NTP1 = G::NTP1, JR = G::JR, JH = G::JH, TP = G::TP;
  constexpr int NLAT = G::NLAT, ROWS = G::ROWS, PITCH = G::PITCH, NCSP = G::NCSP, R = G::R;
  constexpr size_t SPLANE = 2 * (size_t)NCSP;              // floats of a spectral plane (NRSP)
  constexpr size_t FPLANE = (size_t)NLAT * 2 * NTP1;       // floats of a Fourier plane
  constexpr size_t GPLANE = (size_t)NLAT * N;              // floats of a grid plane
  extern __shared__ float4 smem4[];
  float2* tw = reinterpret_cast<float2*>(smem4);
  float2* twq = tw + N;
  float2* fc = twq + 9 * Q;               // [PP][NTP1][PITCH]
  float2* shared = fc + G::PP * G::FC;    // spectral stage [NPAIR][NCSP] float4, or the FFT exchange rows
  float4* spec = reinterpret_cast<float4*>(shared);
  float2* xb = shared;
  float* tab = reinterpret_cast<float*>(shared + G::SHARED);  // [JR][TP]
  int* tpos = reinterpret_cast<int*>(tab + JR * TP);           // [NTP1] first position of m's modes
  const int chunks = JH / JR;
  const int j0 = (blockIdx.x % chunks) * JR;
  // The block's range of passes: the first ranges0 ranges cover the passes
  // below passes0 (the fields with the plain table), the others the rest.
  const int range = blockIdx.x / chunks;
  const bool odd = range >= ranges0;
  const int beg = odd ? passes0 + (range - ranges0) * per_block : range * per_block;
  const int end = min(odd ? set.at[set.n] : passes0, beg + per_block);

  // Spectral coefficients of the pass's plane pairs (p + 2k, p + 2k + 1)
  // as (re a, im a, re b, im b), pair-major.
  float4 rs[R];
  auto fetch = [&](int pass) {
    const int fi = tr_find(set, pass);
    const int p = (pass - set.at[fi]) * G::PP, pend = set.f[fi].planes;
    const float* s = set.f[fi].a;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int e = threadIdx.x + i * G::THREADS;
      const int pair = e / NCSP, w = e - pair * NCSP;
      const int pa = p + 2 * pair;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (e < G::SPEC && pa < pend) {
        const float2 x = reinterpret_cast<const float2*>(s + (size_t)pa * SPLANE)[w];
        const float2 y = pa + 1 < pend ? reinterpret_cast<const float2*>(s + (size_t)(pa + 1) * SPLANE)[w]
                                       : make_float2(0.f, 0.f);
        v = make_float4(x.x, x.y, y.x, y.y);
      }
      rs[i] = v;
    }
  };
  auto store = [&]() {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int e = threadIdx.x + i * G::THREADS;
      if (e < G::SPEC) spec[e] = rs[i];
    }
  };

  {
    // the block's table slice, laid out in HBM as it sits here
    const float4* src = reinterpret_cast<const float4*>((odd ? qj : qi) + (size_t)(j0 / JR) * JR * TP);
    float4* dst = reinterpret_cast<float4*>(tab);
    for (int i = threadIdx.x; i < JR * TP / 4; i += G::THREADS) cp_async16(dst + i, src + i);
  }
  copy_twiddles<Q>(twg, tw, twq);
  if (threadIdx.x == 0) grid_table_positions(NTP1, tpos);
  pdl_wait();
  pdl_release();
  if (beg < end) fetch(beg);
  store();
  cp_async_wait_all();
  __syncthreads();

  const float sg = odd ? -1.f : 1.f;
  const int r = threadIdx.x / T, t = threadIdx.x % T;  // FFT row and lane
  const int pr = r / ROWS, rr = r - pr * ROWS;         // plane of the pass, stage row
  const int lat = stage_lat<G>(rr, j0);
  for (int pass = beg; pass < end; ++pass) {
    const int fi = tr_find(set, pass);
    const int p = (pass - set.at[fi]) * G::PP, pend = set.f[fi].planes, opt = set.f[fi].opt;
    const bool dlambda = (opt & kTrDlambda) != 0;
    // 1. Legendre sums into the coefficient stage.
    {
      const int warp = threadIdx.x / 32, pair = warp / G::WARPS, wi = warp - pair * G::WARPS;
      const int mi = (threadIdx.x % 32) / JR, jj = threadIdx.x % JR;
#pragma unroll 1
      for (int round = 0; round * G::WARPS < G::GROUPS; ++round) {
        const int m = 4 * (round * G::WARPS + ((round & 1) ? G::WARPS - 1 - wi : wi)) + mi;
        if (m >= NTP1) continue;
        const int w0 = mode_start(m, NTP1), K = NTP1 - m;
        const float* qc = tab + jj * TP + tpos[m];
        const float4* sc = spec + pair * NCSP + w0;
        float4 e = make_float4(0.f, 0.f, 0.f, 0.f), o = e;  // (re a, im a, re b, im b)
        int k = 0;
#pragma unroll 2
        for (; k + 1 < K; k += 2) {
          const float qe = qc[k], qo = qc[k + 1];
          const float4 ve = sc[k], vo = sc[k + 1];
          e.x = fmaf(qe, ve.x, e.x);
          e.y = fmaf(qe, ve.y, e.y);
          e.z = fmaf(qe, ve.z, e.z);
          e.w = fmaf(qe, ve.w, e.w);
          o.x = fmaf(qo, vo.x, o.x);
          o.y = fmaf(qo, vo.y, o.y);
          o.z = fmaf(qo, vo.z, o.z);
          o.w = fmaf(qo, vo.w, o.w);
        }
        if (k < K) {
          const float qe = qc[k];
          const float4 ve = sc[k];
          e.x = fmaf(qe, ve.x, e.x);
          e.y = fmaf(qe, ve.y, e.y);
          e.z = fmaf(qe, ve.z, e.z);
          e.w = fmaf(qe, ve.w, e.w);
        }
        float2* fa = fc + (2 * pair) * G::FC + m * PITCH;
        float2* fb = fa + G::FC;
        const int rn = jj, rsouth = ROWS - 1 - jj;
        const float fm = (float)m;
        auto put = [&](float re, float im) { return dlambda ? make_float2(-im * fm, re * fm) : make_float2(re, im); };
        fa[rn] = put(e.x + o.x, e.y + o.y);
        fa[rsouth] = put(sg * (e.x - o.x), sg * (e.y - o.y));
        fb[rn] = put(e.z + o.z, e.w + o.w);
        fb[rsouth] = put(sg * (e.z - o.z), sg * (e.w - o.w));
      }
    }
    __syncthreads();
    if (keep_all || (opt & kTrKeep)) {
      float* f = set.f[fi].x;
      for (int i = threadIdx.x; i < G::PP * NTP1 * ROWS; i += G::THREADS) {
        const int q = i / (NTP1 * ROWS), rem = i - q * NTP1 * ROWS, m = rem / ROWS, row = rem - m * ROWS;
        if (p + q < pend)
          reinterpret_cast<float2*>(f + (size_t)(p + q) * FPLANE)[(size_t)m * NLAT + stage_lat<G>(row, j0)] =
              fc[q * G::FC + m * PITCH + row];
      }
    }
    if (pass + 1 < end) fetch(pass + 1);
    // 2. FFT of the pass's rows (the exchange rows reuse the spectral stage).
    const float2* fr = fc + pr * G::FC;
    float2 a[G::F::QT][8];
#pragma unroll
    for (int i = 0; i < G::F::QT; ++i)
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int k = Q * q + t + T * i, km = M - k;
        float2 gk = k < NTP1 ? fr[k * PITCH + rr] : make_float2(0.f, 0.f);
        if (k == 0) gk.y = 0.f;  // Im c_0 is ignored
        const float2 gmk = conj2(km < NTP1 ? fr[km * PITCH + rr] : make_float2(0.f, 0.f));
        const float2 ev = cadd(gk, gmk);
        const float2 ov = cmul(csub(gk, gmk), tw[k]);
        a[i][q] = make_float2(ev.x - ov.y, ev.y + ov.x);  // e + i o
      }
    float2 b[G::F::KT][Q];
    four_step<Q, 1>(a, b, twq, xb + r * G::F::XP, t);
    if (p + pr < pend) {
      float2* out = reinterpret_cast<float2*>(set.f[fi].y + (size_t)(p + pr) * GPLANE + (size_t)lat * N);
#pragma unroll
      for (int j = 0; j < G::F::KT; ++j)
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2) out[t + T * j + 8 * k2] = b[j][k2];
    }
    __syncthreads();
    if (pass + 1 < end) {
      store();
      __syncthreads();
    }
  }
}

template <int Q, int PP>
void launch_sp2gp(const Model& m, const TrSet& set, cudaStream_t st) {
  using G = GridShape<Q, PP>;
  // the fields with the plain table first
  TrSet s;
  for (int odd = 0; odd < 2; ++odd)
    for (int i = 0; i < set.n; ++i)
      if (((set.f[i].opt & kTrDerivative) != 0) == (odd != 0)) s.add(set.f[i]);
  const int passes = tr_tiles(s, PP);
  int passes0 = passes;
  for (int i = s.n - 1; i >= 0 && (s.f[i].opt & kTrDerivative); --i) passes0 = s.at[i];
  const size_t smem = G::smem();
  const int chunks = G::JH / G::JR;
  const int target = persistent_grid((const void*)k_sp2gp<Q, PP>, G::THREADS, smem);
  const int splits = std::max(1, std::min(passes, (target + chunks - 1) / chunks));
  const int per = (passes + splits - 1) / splits;
  const int ranges0 = (passes0 + per - 1) / per, ranges1 = (passes - passes0 + per - 1) / per;
  step_launch(m.pdl, k_sp2gp<Q, PP>, chunks * (ranges0 + ranges1), G::THREADS, smem, st, s, per, passes0, ranges0,
              m.sh.qiG, m.sh.qjG, reinterpret_cast<const float2*>(m.sh.tw), m.keep_fourier);
}

template <int Q, int PP>
void allow_sp2gp_smem() {
  cudaFuncSetAttribute(k_sp2gp<Q, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GridShape<Q, PP>::smem());
}

}  // namespace

void grid_init() {
  allow_sp2gp_smem<4, 2>();
  allow_sp2gp_smem<8, 2>();
  allow_sp2gp_smem<12, 2>();
  allow_sp2gp_smem<4, 4>();
  allow_sp2gp_smem<8, 4>();
  allow_sp2gp_smem<12, 4>();
}

size_t grid_sp2gp_smem(const Dims& d, int planes_per_pass) {
  const bool four = planes_per_pass == 4;
  switch (d.NLON) {
    case 64: return four ? GridShape<4, 4>::smem() : GridShape<4, 2>::smem();
    case 128: return four ? GridShape<8, 4>::smem() : GridShape<8, 2>::smem();
    default: return four ? GridShape<12, 4>::smem() : GridShape<12, 2>::smem();
  }
}

void grid_sp2gp(const Model& m, const TrSet& s, cudaStream_t st) {
  const bool four = m.tune.sp2gp_planes == 4;
  switch (m.d.NLON) {
    case 64: return four ? launch_sp2gp<4, 4>(m, s, st) : launch_sp2gp<4, 2>(m, s, st);
    case 128: return four ? launch_sp2gp<8, 4>(m, s, st) : launch_sp2gp<8, 2>(m, s, st);
    default: return four ? launch_sp2gp<12, 4>(m, s, st) : launch_sp2gp<12, 2>(m, s, st);
  }
}

}  // namespace exogcm
