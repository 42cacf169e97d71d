// Host side of the two-pass stage (fft_flex.cuh): which lengths it takes, and
// the launch.
#include <algorithm>
#include <map>

#include "fft_flex.cuh"
#include "fft_flex_lengths.h"

namespace dfft {
namespace dev {

using namespace flex;

namespace {

struct Split {
  int m, r1, r2;
};
#define DFFT_SPLIT(M_, R1_, R2_) {M_, R1_, R2_},
const Split kPlain[] = {DFFT_FLEX_PLAIN_0(DFFT_SPLIT) DFFT_FLEX_PLAIN_1(DFFT_SPLIT) DFFT_FLEX_PLAIN_2(DFFT_SPLIT)
                            DFFT_FLEX_PLAIN_3(DFFT_SPLIT) DFFT_FLEX_PLAIN_4(DFFT_SPLIT) DFFT_FLEX_PLAIN_5(DFFT_SPLIT)
                                DFFT_FLEX_PLAIN_6(DFFT_SPLIT) DFFT_FLEX_PLAIN_7(DFFT_SPLIT)};
const Split kChirp[] = {DFFT_FLEX_CHIRP_0(DFFT_SPLIT) DFFT_FLEX_CHIRP_1(DFFT_SPLIT) DFFT_FLEX_CHIRP_2(DFFT_SPLIT)
                            DFFT_FLEX_CHIRP_3(DFFT_SPLIT)};
#undef DFFT_SPLIT

template <typename T, bool CHIRP, int... G>
std::map<int, Entry> all_entries() {
  std::map<int, Entry> all;
  auto add = [&](const Entry* (*get)(int*)) {
    int n = 0;
    const Entry* e = get(&n);
    for (int i = 0; i < n; ++i) all[e[i].m] = e[i];
  };
  (add(&Group<T, CHIRP, G>::entries), ...);
  return all;
}

const Entry* find_entry(bool dbl, bool chirp, int m) {
  static const std::map<int, Entry> tables[4] = {
      all_entries<float, false, 0, 1, 2, 3, 4, 5, 6, 7>(), all_entries<float, true, 0, 1, 2, 3>(),
      all_entries<double, false, 0, 1, 2, 3, 4, 5, 6, 7>(), all_entries<double, true, 0, 1, 2, 3>()};
  const auto& t = tables[(dbl ? 2 : 0) + (chirp ? 1 : 0)];
  const auto it = t.find(m);
  return it == t.end() ? nullptr : &it->second;
}

}  // namespace

bool flex_split(int m, bool chirp, int* R1, int* R2) {
  auto find = [&](const Split* s, const Split* end) {
    const Split* f = std::find_if(s, end, [&](const Split& x) { return x.m == m; });
    if (f == end) return false;
    *R1 = f->r1;
    *R2 = f->r2;
    return true;
  };
  return chirp ? find(std::begin(kChirp), std::end(kChirp)) : find(std::begin(kPlain), std::end(kPlain));
}

// The shortest length of the table that is at least 2 n - 1 and 5/8 of the
// power of two that is.  A convolution's rounding errors spread over its m
// points, of which the line keeps n: error = q sqrt(n / m), q within 3 % the
// same for all n: 2.1e-7 to 2.5e-7 (complex64) and 3.6e-16 to 4.6e-16
// (complex128) for the splits listed, 2.5e-7 to 3.1e-7 and 4.0e-16 to 5.6e-16
// for powers of two in register passes, more for splits with 9, 18, 25 or 27.
// Against the power of two, over the 343 lengths up to 512: errors 0.98 times
// as large on average, at most 1.06 (complex64) and 1.12 (complex128); with the
// shortest 5-smooth length 1.04 and 1.07, at most 1.21 and 1.51.
int flex_chirp_length(int n) {
  int power = 1, best = 0;
  while (power < 2 * n - 1) power *= 2;
  for (const Split& s : kChirp)
    if (s.m >= 2 * n - 1 && 8 * s.m >= 5 * power && (best == 0 || s.m < best)) best = s.m;
  return best;
}

int flex_lines(bool dbl, bool afast, int R1) {
  return dbl ? tile_lines<double>(afast, R1) : tile_lines<float>(afast, R1);
}

cudaError_t launch_fft_flex(const StageArgs& A, const FlexArgs& F0, bool dbl, int kind, bool inverse,
                            cudaStream_t st) {
  if (A.Eo0 > fast_stage_max_grid_yz() || A.Eo1 > fast_stage_max_grid_yz()) return cudaErrorInvalidValue;
  const Entry* e = find_entry(dbl, F0.chirp != nullptr, F0.m);
  if (!e) return cudaErrorInvalidValue;
  FlexArgs F = F0;
  F.inverse = inverse ? 1 : 0;
  const bool af = A.load_afast != 0;
  LaunchFn fn = nullptr;
  if (kind == kC2C)
    fn = af ? e->c2c_a : e->c2c_b;
  else if (kind == kR2C && af)
    fn = e->r2c;
  else if (kind == kC2R && af)
    fn = e->c2r;
  return fn ? fn(A, F, st) : cudaErrorInvalidValue;
}

}  // namespace dev
}  // namespace dfft
