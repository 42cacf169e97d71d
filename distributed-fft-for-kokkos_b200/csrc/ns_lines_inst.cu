// One group of instantiations of the Navier-Stokes line kernels
// (ns_lines.cuh), chosen by the build: NSL_T (float, double), NSL_GROUP and
// NSL_LIST, a group of ns_lengths.h and its macro.
#include "ns_lengths.h"
#include "ns_lines.cuh"

namespace dfft {
namespace dev {
namespace nsl {

namespace {

template <typename T, int KIND, int R1, int R2>
cudaError_t launch_line(const LineArgs<T>& a, int nf, cudaStream_t st) {
  using S = LineShape<T, R1, R2>;
  auto k = ns_line_kernel<T, KIND, R1, R2>;
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k), S::smem);
  if (e != cudaSuccess) return e;
  const dim3 grid(static_cast<unsigned>((a.lines + S::B - 1) / S::B), 3, static_cast<unsigned>(nf));
  const size_t bytes = sizeof(cplx<T>) * R1 * R2 * a.lines * 3 * nf;
  return launch_kernel_early(bytes <= kEarlyStartBytes, k, grid, S::NT, S::smem, st, a);
}

template <typename T, int R1, int R2, bool ADJ>
cudaError_t launch_z(const ZArgs<T>& a, cudaStream_t st) {
  using S = ZShape<T, R1, R2, ADJ>;
  if constexpr (S::ok) {
    auto k = ns_z_kernel<T, R1, R2, ADJ>;
    const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k), S::smem);
    if (e != cudaSuccess) return e;
    const int pairs = (a.points + 1) / 2;
    const size_t bytes = sizeof(cplx<T>) * 9 * a.points * a.g.z.k;
    return launch_kernel_early(bytes <= kEarlyStartBytes, k, dim3(static_cast<unsigned>((pairs + S::G - 1) / S::G)), S::NT,
                               S::smem, st, a);
  } else {
    return cudaErrorInvalidValue;
  }
}

template <typename T, int R1, int R2>
constexpr Entry<T> entry() {
  return Entry<T>{R1 * R2, R1, R2,
                  {launch_line<T, kXInverse, R1, R2>, launch_line<T, kYInverse, R1, R2>,
                   launch_line<T, kYForward, R1, R2>, launch_line<T, kXForward, R1, R2>},
                  ZShape<T, R1, R2, false>::ok ? launch_z<T, R1, R2, false> : nullptr,
                  ZShape<T, R1, R2, true>::ok ? launch_z<T, R1, R2, true> : nullptr};
}

}  // namespace

template <>
const Entry<NSL_T>* Group<NSL_T, NSL_GROUP>::entries(int* count) {
  static const Entry<NSL_T> list[] = {
#define DFFT_ENTRY(N_, R1_, R2_) entry<NSL_T, R1_, R2_>(),
      NSL_LIST(DFFT_ENTRY)
#undef DFFT_ENTRY
  };
  *count = static_cast<int>(sizeof(list) / sizeof(list[0]));
  return list;
}

}  // namespace nsl
}  // namespace dev
}  // namespace dfft
