// One group of instantiations of the two-pass stage (fft_flex.cuh), chosen by
// the build: FLEX_T (float, double), FLEX_CLS (0, 1, 2), FLEX_CHIRP (false,
// true).  A group per translation unit, so that they compile side by side.
#include "fft_flex.cuh"

namespace dfft {
namespace dev {
namespace flex {

template <>
cudaError_t launch_class<FLEX_T, FLEX_CLS, FLEX_CHIRP>(const StageArgs& A, const FlexArgs& F, int kind,
                                                       cudaStream_t st) {
  const bool af = A.load_afast != 0;
  if (kind == kC2C)
    return af ? launch_kernel<FLEX_T, kC2C, true, FLEX_CLS, FLEX_CHIRP>(A, F, st)
              : launch_kernel<FLEX_T, kC2C, false, FLEX_CLS, FLEX_CHIRP>(A, F, st);
  if (!af) return cudaErrorInvalidValue;
  if (kind == kR2C) return launch_kernel<FLEX_T, kR2C, true, FLEX_CLS, FLEX_CHIRP>(A, F, st);
  if (kind == kC2R) return launch_kernel<FLEX_T, kC2R, true, FLEX_CLS, FLEX_CHIRP>(A, F, st);
  return cudaErrorInvalidValue;
}

}  // namespace flex
}  // namespace dev
}  // namespace dfft
