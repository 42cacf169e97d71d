// Host side of the two-pass stage (fft_flex.cuh): which lengths it takes, its
// tiles, and the launch.
#include <algorithm>

#include "fft_flex.cuh"

namespace dfft {
namespace dev {

using namespace flex;

namespace {

#define DFFT_OK(R_) case R_:
bool small_codelet(int r) {
  switch (r) {
    DFFT_FLEX_R1(DFFT_OK) return true;
    default: return false;
  }
}
bool large_codelet(int r) {
  switch (r) {
    DFFT_FLEX_R2(DFFT_OK) return true;
    default: return false;
  }
}
#undef DFFT_OK
// both radices in one register class's kernels
bool codelet_pair(int a, int b) { return (small_codelet(a) && small_codelet(b)) || (large_codelet(a) && large_codelet(b)); }

unsigned magic(int d) { return static_cast<unsigned>(((1ull << 32) + d - 1) / d); }

}  // namespace

// The most even split: the kernel's registers (and so its resident threads)
// follow the larger codelet.
bool flex_split(int m, int* R1, int* R2) {
  int best = 0;
  for (int r2 = 2; r2 * r2 <= m; ++r2)
    if (m % r2 == 0 && codelet_pair(m / r2, r2)) best = r2;
  if (best == 0) return false;
  *R1 = m / best;
  *R2 = best;
  return true;
}

// The smallest m >= 2n - 1 that splits into codelets without a factor 11 or
// 13 (those codelets cost O(R^2) operations).
int flex_chirp_length(int n) {
  for (int m = 2 * n - 1; m <= 32 * 32; ++m) {
    int r1 = 0, r2 = 0;
    if (m % 11 != 0 && m % 13 != 0 && flex_split(m, &r1, &r2)) return m;
  }
  return 0;
}

// Options: bit 0 swaps the radices (a-fast rows are read in runs of R2 and
// written in runs of R1 elements), bit 1 halves the tile.  Tiles: a-fast about
// 256 complex64 or 192 complex128 butterflies; b-fast rows of 128 bytes.
bool flex_config(bool dbl, int kind, bool afast, int n, int m, int opt, FlexArgs* F) {
  if (kind != kC2C && !afast) return false;
  if (opt < 0 || opt >= kFlexOptions) return false;
  const bool chirp = m != n;
  int r1 = 0, r2 = 0;
  if (!flex_split(m, &r1, &r2)) return false;
  if ((opt & 1) && r1 == r2) return false;
  *F = FlexArgs{};
  F->n = n;
  F->m = m;
  F->R1 = (opt & 1) ? r2 : r1;
  F->R2 = (opt & 1) ? r1 : r2;
  F->cls = r1 <= 10 ? 0 : r1 <= 16 ? 1 : 2;
  const size_t ce = dbl ? 16 : 8;
  const int odd1 = F->R1 | 1, odd2 = F->R2 | 1;
  F->P0 = afast ? F->R2 * odd1 : m;
  F->P1 = chirp ? (afast ? F->R1 * odd2 : m) : 0;
  const int zn = afast ? (n | 1) : n;
  if (kind == kC2R || (kind == kR2C && !chirp)) F->P1 = std::max(F->P1, zn);
  if (kind == kR2C && chirp) F->P0 = std::max(F->P0, zn);
  const int most = std::max(F->R1, F->R2);
  int B = afast ? std::max(1, (dbl ? 192 : 256) / most) : (dbl ? 8 : 16);
  if (opt & 2) {
    if (B < 2) return false;
    B /= 2;
  }
  const size_t line = (static_cast<size_t>(F->P0) + F->P1) * ce;
  while (B > 1 && line * B > 100 * 1024) B /= 2;
  if (line * B > 227 * 1024) return false;
  F->B = B;
  F->smem = line * B;
  if (!afast)
    while ((1 << F->lshift) < B) ++F->lshift;
  const int total = B * most, cap = dbl ? 256 : 512;
  const int loops = (total + cap - 1) / cap;
  F->nthreads = std::min(cap, ((total + loops - 1) / loops + 31) / 32 * 32);
  F->share = F->nthreads / B;
  if (F->share < 2) return false;
  F->magic1 = magic(F->R1);
  F->magic2 = magic(F->R2);
  F->magic_share = magic(F->share);
  return true;
}

namespace flex {
#define DFFT_DECL(T, CLS, CHIRP) \
  template <>                    \
  cudaError_t launch_class<T, CLS, CHIRP>(const StageArgs& A, const FlexArgs& F, int kind, cudaStream_t st);
DFFT_DECL(float, 0, false) DFFT_DECL(float, 1, false) DFFT_DECL(float, 2, false)
DFFT_DECL(float, 0, true) DFFT_DECL(float, 1, true) DFFT_DECL(float, 2, true)
DFFT_DECL(double, 0, false) DFFT_DECL(double, 1, false) DFFT_DECL(double, 2, false)
DFFT_DECL(double, 0, true) DFFT_DECL(double, 1, true) DFFT_DECL(double, 2, true)
#undef DFFT_DECL

template <typename T, bool CHIRP>
static cudaError_t launch_any_class(const StageArgs& A, const FlexArgs& F, int kind, cudaStream_t st) {
  switch (F.cls) {
    case 0: return launch_class<T, 0, CHIRP>(A, F, kind, st);
    case 1: return launch_class<T, 1, CHIRP>(A, F, kind, st);
    case 2: return launch_class<T, 2, CHIRP>(A, F, kind, st);
    default: return cudaErrorInvalidValue;
  }
}
}  // namespace flex

cudaError_t launch_fft_flex(const StageArgs& A, const FlexArgs& F0, bool dbl, int kind, bool inverse,
                            cudaStream_t st) {
  if (A.Eo0 > fast_stage_max_grid_yz() || A.Eo1 > fast_stage_max_grid_yz()) return cudaErrorInvalidValue;
  FlexArgs F = F0;
  F.swap = (kind == kC2C && inverse) ? 1 : 0;
  if (F.chirp)
    return dbl ? launch_any_class<double, true>(A, F, kind, st) : launch_any_class<float, true>(A, F, kind, st);
  return dbl ? launch_any_class<double, false>(A, F, kind, st) : launch_any_class<float, false>(A, F, kind, st);
}

}  // namespace dev
}  // namespace dfft
