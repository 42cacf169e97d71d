// Kernels of the batched register stages (see fft_batch.cu): the tile bodies
// of fft_tile.cuh behind a work table.  Instantiated for
// general-layout sides (AFF, fft_batch.cu) and separable sides only
// (fft_batch_sep.cu, fewer registers) in two translation units.
#pragma once

#include <cstring>

#include "fft_fast.cuh"
#include "fft_pair.cuh"

namespace dfft {
namespace dev {
namespace batch {

using namespace radix;


// A launch covers the fields of one line length N, one tile per CTA, so each
// kernel carries one tile body at the register budget of its one-field kernel
// (MinBlocks of fft_fast.cuh).  Lines per tile: 256 threads for 8-value bodies;
// 128 for 24-value ones where that leaves 128-byte rows (16 complex64 or 8
// complex128), else 256.  (Persistent CTAs of 256 threads that walked the work
// table held the 24-value bodies to 512 threads per SM, two CTAs waiting at
// their barriers: 132 us a stage of five 192^3 complex64 fields.)
template <typename T, int N>
struct BatchLines {
  static constexpr int tt = N / Vals<N>::value;  // threads a line
  static constexpr int rows = sizeof(T) == 4 ? 16 : 8;
  static constexpr int threads = Vals<N>::value == 24 && rows * tt <= 128 ? 128 : 256;
  static constexpr int value = threads / tt;
};

#define DFFT_BATCH_LENGTHS(X) \
  X(16) X(32) X(64) X(128) X(256) X(512) X(1024) X(2048) X(24) X(48) X(96) X(192) X(384) X(768)

// tile (tb, co0, co1) of a field's stage from its local work index (32-bit:
// the host keeps every field's tile count below 2^31)
__device__ __forceinline__ void decode(const StageArgs& A, unsigned local, int* tb, int* co0, int* co1) {
  const unsigned tbs = static_cast<unsigned>(A.tiles_b);
  *tb = static_cast<int>(local % tbs);
  const unsigned rest = local / tbs;
  *co0 = static_cast<int>(rest % static_cast<unsigned>(A.Eo0));
  *co1 = static_cast<int>(rest / static_cast<unsigned>(A.Eo0));
}

// the field and tile of work item w: the fields of a launch follow one another
__device__ __forceinline__ const StageArgs& locate(const BatchParams& P, long long w, int* tb, int* co0, int* co1) {
  int f = 0;
  while (w >= P.prefix[f + 1]) ++f;
  decode(P.f[f], static_cast<unsigned>(w - P.prefix[f]), tb, co0, co1);
  return P.f[f];
}

template <typename T, bool INV, bool AFAST, bool AFF, int N>
__global__ void __launch_bounds__((BatchLines<T, N>::threads), (MinBlocks<T, N, BatchLines<T, N>::threads, AFAST, AFF>::value))
    fft_batch_c2c_kernel(const __grid_constant__ BatchParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  release_dependents();
  int tb, co0, co1;
  const StageArgs& A = locate(P, blockIdx.x, &tb, &co0, &co1);
  fast_tile<T, INV, N, BatchLines<T, N>::value, AFAST, AFF>(A, tb, co0, co1, smem_raw);
}

template <typename T, bool C2R, bool AFF, int N>
__global__ void __launch_bounds__((BatchLines<T, N>::threads), (MinBlocks<T, N, BatchLines<T, N>::threads, true, AFF>::value))
    fft_batch_real_kernel(const __grid_constant__ BatchParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  release_dependents();
  int tb, co0, co1;
  const StageArgs& A = locate(P, blockIdx.x, &tb, &co0, &co1);
  real_tile<T, C2R, N, BatchLines<T, N>::value, AFF>(A, tb, co0, co1, smem_raw);
}

// Two-line (complex64, separable, 2^k points) batched C2C stage: the tile
// body of fft_pair_kernel with its default pairs per tile, N/8 threads per
// pair, at that kernel's register budget (1024 resident threads per SM).
template <int N, bool AFAST>
struct BatchPairs {
  static constexpr int value = pair_option(N, AFAST, 0);
  static constexpr int threads = N / 8 * value;
  static constexpr int min_blocks = 1024 / threads > 0 ? 1024 / threads : 1;
};

template <bool INV, bool AFAST, int N>
__global__ void __launch_bounds__(BatchPairs<N, AFAST>::threads, (BatchPairs<N, AFAST>::min_blocks))
    fft_batch_pair_kernel(const __grid_constant__ BatchParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  release_dependents();
  int tb, co0, co1;
  const StageArgs& A = locate(P, blockIdx.x, &tb, &co0, &co1);
  pair_tile<INV, N, BatchPairs<N, AFAST>::value, AFAST>(A, tb, co0, co1, smem_raw);
}

template <typename T>
size_t tile_smem(int n, bool afast) {
  switch (n) {
#define DFFT_SMEM(N_)                                                                                        \
  case N_:                                                                                                   \
    return sizeof(cplx<T>) * (N_ + static_cast<size_t>(BatchLines<T, N_>::value) *                              \
                                       (afast ? SmemShape<T, N_, BatchLines<T, N_>::value, true>::LP         \
                                              : SmemShape<T, N_, BatchLines<T, N_>::value, false>::LP));
    DFFT_BATCH_LENGTHS(DFFT_SMEM)
#undef DFFT_SMEM
    default: return 0;
  }
}

template <typename C, int THREADS, typename K>
cudaError_t launch_tiles(K kernel, const BatchParams& P, size_t smem, cudaStream_t st) {
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(kernel), smem);
  if (e != cudaSuccess) return e;
  const long long total = P.prefix[P.nfields];
  if (total < 1) return cudaSuccess;
  if (total >= (1ll << 31)) return cudaErrorInvalidConfiguration;
  return launch_kernel_early(early_start(P, sizeof(C)), kernel, dim3(static_cast<unsigned>(total)), THREADS, smem, st, P);
}

template <bool INV, bool AFAST, int N>
cudaError_t launch_batch_pair_n(BatchParams& P, cudaStream_t st) {
  constexpr size_t smem = pair_tile_smem<N, BatchPairs<N, AFAST>::value, AFAST>();
  for (int i = 0; i < P.nfields; ++i) P.f[i] = with_table_offsets(P.f[i]);
  return launch_tiles<float2, BatchPairs<N, AFAST>::threads>(fft_batch_pair_kernel<INV, AFAST, N>, P, smem, st);
}

template <typename T, bool AFF, int N>
cudaError_t launch_batch_n(BatchParams& P, size_t smem, int kind, bool inverse, bool afast, cudaStream_t st) {
  constexpr int NT = BatchLines<T, N>::threads;
  if (kind == kC2C) {
    if (inverse)
      return afast ? launch_tiles<cplx<T>, NT>(fft_batch_c2c_kernel<T, true, true, AFF, N>, P, smem, st)
                   : launch_tiles<cplx<T>, NT>(fft_batch_c2c_kernel<T, true, false, AFF, N>, P, smem, st);
    return afast ? launch_tiles<cplx<T>, NT>(fft_batch_c2c_kernel<T, false, true, AFF, N>, P, smem, st)
                 : launch_tiles<cplx<T>, NT>(fft_batch_c2c_kernel<T, false, false, AFF, N>, P, smem, st);
  }
  if (kind == kR2C) return launch_tiles<cplx<T>, NT>(fft_batch_real_kernel<T, false, AFF, N>, P, smem, st);
  if (kind == kC2R) return launch_tiles<cplx<T>, NT>(fft_batch_real_kernel<T, true, AFF, N>, P, smem, st);
  return cudaErrorInvalidValue;
}

// every field of P has the same line length (the host groups them)
template <typename T, bool AFF>
cudaError_t launch_batch_t(BatchParams& P, int kind, bool inverse, bool afast, cudaStream_t st) {
  const int n = P.f[0].n;
  const size_t smem = tile_smem<T>(n, kind == kC2C ? afast : true);
  if (smem == 0) return cudaErrorInvalidValue;
  for (int i = 0; i < P.nfields; ++i) {
    if (P.f[i].n != n) return cudaErrorInvalidValue;
    P.f[i] = with_table_offsets(P.f[i]);
  }
  switch (n) {
#define DFFT_LAUNCH(N_) \
  case N_: return launch_batch_n<T, AFF, N_>(P, smem, kind, inverse, afast, st);
    DFFT_BATCH_LENGTHS(DFFT_LAUNCH)
#undef DFFT_LAUNCH
    default: return cudaErrorInvalidValue;
  }
}

// the launcher of one addressing variant (AFF: general-layout sides),
// defined in fft_batch.cu (AFF = true) and fft_batch_sep.cu (AFF = false)
template <bool AFF>
cudaError_t launch_batch_variant(BatchParams& P, bool dbl, int kind, bool inverse, bool afast, cudaStream_t st);
template <>
cudaError_t launch_batch_variant<true>(BatchParams& P, bool dbl, int kind, bool inverse, bool afast, cudaStream_t st);
template <>
cudaError_t launch_batch_variant<false>(BatchParams& P, bool dbl, int kind, bool inverse, bool afast, cudaStream_t st);

}  // namespace batch
}  // namespace dev
}  // namespace dfft
