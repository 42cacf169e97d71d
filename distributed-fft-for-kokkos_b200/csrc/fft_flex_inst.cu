// One group of instantiations of the two-pass stage (fft_flex.cuh), chosen by
// the build: FLEX_T (float, double), FLEX_CHIRP (false, true) FLEX_GROUP and
// FLEX_LIST, a group of fft_flex_lengths.h and its macro.
#include "fft_flex.cuh"
#include "fft_flex_lengths.h"

namespace dfft {
namespace dev {
namespace flex {

template <>
const Entry* Group<FLEX_T, FLEX_CHIRP, FLEX_GROUP>::entries(int* count) {
  static const Entry list[] = {
#define DFFT_ENTRY(M_, R1_, R2_)                                                                          \
  {M_, launch_kernel<FLEX_T, kC2C, true, R1_, R2_, FLEX_CHIRP>,                                           \
   launch_kernel<FLEX_T, kC2C, false, R1_, R2_, FLEX_CHIRP>,                                              \
   launch_kernel<FLEX_T, kR2C, true, R1_, R2_, FLEX_CHIRP>, launch_kernel<FLEX_T, kC2R, true, R1_, R2_, FLEX_CHIRP>},
      FLEX_LIST(DFFT_ENTRY)
#undef DFFT_ENTRY
  };
  *count = static_cast<int>(sizeof(list) / sizeof(list[0]));
  return list;
}

}  // namespace flex
}  // namespace dev
}  // namespace dfft
