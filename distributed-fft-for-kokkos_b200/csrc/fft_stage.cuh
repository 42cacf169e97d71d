// Device helpers shared by the .cu translation units.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "dev_types.h"

namespace dfft {
namespace dev {

template <typename T> struct CplxOf;
template <> struct CplxOf<float> { using type = float2; };
template <> struct CplxOf<double> { using type = double2; };
template <typename T> using cplx = typename CplxOf<T>::type;

template <typename T> __device__ __forceinline__ cplx<T> mk(T x, T y) { cplx<T> r; r.x = x; r.y = y; return r; }
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  C r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
template <typename C, typename T> __device__ __forceinline__ C cscale(C a, T s) { C r; r.x = a.x * s; r.y = a.y * s; return r; }
// a + s b
template <typename C, typename T> __device__ __forceinline__ C cfma(C b, T s, C a) { C r; r.x = a.x + s * b.x; r.y = a.y + s * b.y; return r; }
template <typename C> __device__ __forceinline__ C cconj(C a) { a.y = -a.y; return a; }
// s*i*z with s = -1 for the forward transform and +1 for the inverse.
template <bool INV, typename C> __device__ __forceinline__ C rot(C z) {
  C r;
  if (INV) { r.x = -z.y; r.y = z.x; } else { r.x = z.y; r.y = -z.x; }
  return r;
}

// a + rot(z), a - rot(z): without the rotated value
template <bool INV, typename C> __device__ __forceinline__ C cadd_rot(C a, C z) {
  C r;
  if (INV) { r.x = a.x - z.y; r.y = a.y + z.x; } else { r.x = a.x + z.y; r.y = a.y - z.x; }
  return r;
}
template <bool INV, typename C> __device__ __forceinline__ C csub_rot(C a, C z) { return cadd_rot<!INV>(a, z); }
// a + s rot(z)
template <bool INV, typename C, typename T> __device__ __forceinline__ C cfma_rot(C z, T s, C a) {
  C r;
  if (INV) { r.x = a.x - s * z.y; r.y = a.y + s * z.x; } else { r.x = a.x + s * z.y; r.y = a.y - s * z.x; }
  return r;
}

// complex64: both parts in one packed instruction (sm_100 add / mul / fma
// .f32x2, each part rounded as the scalar instruction does).  The radix passes
// are bound by instruction issue as much as by memory, and additions of whole
// values are most of their arithmetic; rotated operands and complex products
// stay scalar (packed forms of them need moves), and products that are added
// to go through cfma, one rounding as before.  Two-pass stages of 300 x 250 x
// 360: 97, 86 and 86 -> 86, 83 and 81 us; Navier-Stokes z lines at 192^3: 162
// -> 154 us.
__device__ __forceinline__ unsigned long long pack2(float2 v) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v.x), "f"(v.y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(r);
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(r);
}
__device__ __forceinline__ float2 cscale(float2 a, float s) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(make_float2(s, s))));
  return unpack2(r);
}
__device__ __forceinline__ float2 cfma(float2 b, float s, float2 a) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack2(b)), "l"(pack2(make_float2(s, s))), "l"(pack2(a)));
  return unpack2(r);
}

// Programmatic dependent launch.  A kernel launched with `early` may start
// while the one before it in the stream drains: it stages tables and computes
// addresses (nothing another kernel writes), then waits in dependency_wait for
// that kernel's completion before it touches data.  release_dependents, at the
// top of a kernel, lets the next one start so as soon as every CTA of this one
// is running.  In a kernel launched the plain way both return at once.
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Early starts pay for short kernels, whose launch gap and prologue show: 32^3
// complex128 24.6 -> 20.3 us for six stages of 0.5 MB, 256 x 192 x 128
// complex64 93.7 -> 82.3 us for four of 50 MB.  Past that a stage has waves
// enough that the waiting CTAs only disturb its end: six stages of 1 GB ran in
// 2861 us with early starts and 2490 us without, 216 MB ones in 565 and 555.
constexpr size_t kEarlyStartBytes = size_t(128) << 20;

template <typename... P, typename... Args>
inline cudaError_t launch_kernel_early(bool early, void (*kernel)(P...), dim3 grid, int threads, size_t smem,
                                       cudaStream_t st, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  if (e != cudaSuccess) cudaGetLastError();  // reported here, not by the next launch's check
  return e;
}

// a launch's early start: by the bytes of the arrays it reads (complex elements)
inline size_t stage_bytes(const StageArgs& A, size_t elem) { return static_cast<size_t>(A.n) * A.Eb * A.Eo0 * A.Eo1 * elem; }
inline bool early_start(const StageArgs& A, size_t elem) {
  return !A.plain_launch && stage_bytes(A, elem) <= kEarlyStartBytes;
}
inline bool early_start(const BatchParams& P, size_t elem) {
  size_t bytes = 0;
  bool plain = false;
  for (int i = 0; i < P.nfields; ++i) {
    bytes += stage_bytes(P.f[i], elem);
    plain = plain || P.f[i].plain_launch;
  }
  return !plain && bytes <= kEarlyStartBytes;
}

// Element offset of global coordinate c (nd axes) in a layout.
__device__ __forceinline__ int64_t layout_offset(const DevLayout& L, const int* c, int nd) {
  if (L.mode == 0) {
    int64_t o = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < nd) o += __ldg(L.t + L.off[k] + c[k]);
    return o;
  }
  int64_t r = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (k < nd) r += __ldg(L.t + L.rk[k] + c[k]);
  int64_t o = __ldg(L.t + L.rbase + r);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (k < nd) o += __ldg(L.t + L.loc[k] + c[k]) * __ldg(L.t + L.rstride + r * 4 + k);
  return o;
}

}  // namespace dev
}  // namespace dfft
