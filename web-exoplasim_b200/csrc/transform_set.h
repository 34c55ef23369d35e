// The fields of one transform launch.
#pragma once
#include <stdexcept>

namespace exogcm {

// A set of fields one transform launch works through: independent planes of
// several fields in one grid, so that a step pays one launch, one ramp and
// one tail for all of them. What the pointers mean is each transform's own.
struct TrField {
  const float* a = nullptr;
  const float* b = nullptr;
  const float* c = nullptr;
  float* x = nullptr;
  float* y = nullptr;
  int planes = 0;
  int opt = 0;
  float plavor = 0.f;
};
constexpr int kMaxTr = 12;
struct TrSet {
  int n = 0;
  int at[kMaxTr + 1] = {};  // first tile of each field (tr_tiles)
  TrField f[kMaxTr];
  void add(const TrField& t) {
    if (n == kMaxTr) throw std::logic_error("transform launch: too many fields");
    f[n++] = t;
  }
};
// Numbers the tiles of `tile` planes of the set's fields one after another
// (no tile spans two fields); returns their count.
inline int tr_tiles(TrSet& s, int tile) {
  s.at[0] = 0;
  for (int i = 0; i < s.n; ++i) s.at[i + 1] = s.at[i] + (s.f[i].planes + tile - 1) / tile;
  return s.at[s.n];
}
// Whether the set's fields are of a kind, for launches that take one kind at a
// time: every field or none.
template <typename F>
bool tr_every(const TrSet& s, F of_kind) {
  const bool first = s.n > 0 && of_kind(s.f[0]);
  for (int i = 1; i < s.n; ++i)
    if (of_kind(s.f[i]) != first) throw std::logic_error("transform launch: fields of two kinds");
  return first;
}
#ifdef __CUDACC__
// The field of a tile; tile - s.at[field] is the tile's number in it.
__device__ __forceinline__ int tr_find(const TrSet& s, int tile) {
  int f = 0;
  while (f + 1 < s.n && tile >= s.at[f + 1]) ++f;
  return f;
}
#endif

// Options of a spectral -> grid field (TrField::opt).
constexpr int kTrDerivative = 1;  // sp2fcdmu: the d/dmu table
constexpr int kTrDlambda = 2;     // d/dlambda of the Fourier coefficients before fc2gp
constexpr int kTrKeep = 4;        // the Fourier field is written whatever Model::keep_fourier

}  // namespace exogcm
