// Two-pass FFT stage for lines of m = R1 R2 points, R1 and R2 any two codelet
// lengths up to 32 (sm_100a): every 2^a 3^b 5^c 7^d 11^e 13^f length up to
// about 700 that splits so, and, through the chirp-z convolution, every other
// length n whose 2 n - 1 fits such an m.
//
// What bounds it: bytes.  A tile of B lines is read from global memory once
// and written once; between the two passes a line crosses shared memory once
// (chirp-z: twice).  Pass 1 gives every thread an R1-point codelet whose inputs
// it loads itself, R1 independent loads in flight per thread; it leaves row j
// of the line's R2 x R1 matrix in shared memory; pass 2 reads columns, applies
// the twiddle w_m^(j r) and stores straight to global memory.  So there is one
// barrier between loads and stores, and the CTAs of an SM, each at a different
// point, keep the memory busy.
//
// Measured (B200, forward + backward transform, before: the table-driven
// shared-memory kernel of fft_stage.cu, chirp-z as five launches): 300 x 250 x
// 360 complex64 3816 -> 810 us, 200 x 180 x 252 R2C / C2R double 1633 -> 467 us,
// 131 x 105 x 157 R2C / C2R double 768 -> 331 us.
//
// The radices are run-time values (a switch over compile-time codelets), one
// kernel per register class: codelets up to 10, 16 and 32 points.
//
// Thread mapping: a-fast rows (unit stride along the FFT axis) take the
// butterflies of a line on consecutive threads, with the matrix rows padded
// to an odd pitch; b-fast rows (unit stride along the tile axis) take the B
// lines of a tile on consecutive threads.
#pragma once

#include "fft_codelet.cuh"

namespace dfft {
namespace dev {
namespace flex {

using codelet::Dft;

template <typename T, int CLS>
struct Bounds {
  // complex64: 512 threads (128 registers); complex128: 256 threads, two CTAs
  // (128 registers) up to 16-point codelets, one (255 registers) above
  static constexpr bool f32 = sizeof(T) == 4;
  static constexpr int threads = f32 ? 512 : 256;
  static constexpr int blocks = f32 ? 1 : (CLS < 2 ? 2 : 1);
};

// positions of a line: affine, or from the axis table
struct Line {
  int64_t base, stride;
  const int64_t* tab;
  __device__ __forceinline__ int64_t at(int p) const { return base + (tab ? __ldg(tab + p) : p * stride); }
};

// f(r, offset of position p0 + r * step) for r < R with p0 + r * step < lim
// (LIM: else every r); one affine or one table loop, no choice per element
template <int R, bool LIM, typename Fn>
__device__ __forceinline__ void each(const Line& l, int p0, int step, int lim, Fn&& f) {
  if (l.tab) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (!LIM || p0 + r * step < lim) f(r, l.base + __ldg(l.tab + p0 + r * step));
  } else {
    const int64_t b = l.base + p0 * l.stride, st = step * l.stride;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (!LIM || p0 + r * step < lim) f(r, b + r * st);
  }
}

__device__ __forceinline__ Line src_line(const StageArgs& A, int lb, int co0, int co1) {
  Line l;
  l.tab = nullptr;
  if (A.src_line_affine) {
    radix::line_affine(A.src, A, lb, co0, co1, &l.base, &l.stride);
    return l;
  }
  l.base = A.src_abase + __ldg(A.src.t + A.s_tb + lb);
  if (A.o0 >= 0) l.base += __ldg(A.src.t + A.s_to0 + co0);
  if (A.o1 >= 0) l.base += __ldg(A.src.t + A.s_to1 + co1);
  l.stride = A.src_astride;
  if (A.src_atab) l.tab = A.src.t + A.s_ta;
  return l;
}

__device__ __forceinline__ Line dst_line(const StageArgs& A, int lb, int co0, int co1) {
  Line l;
  l.tab = nullptr;
  if (A.dst_line_affine) {
    radix::line_affine(A.dst, A, lb, co0, co1, &l.base, &l.stride);
    return l;
  }
  l.base = A.dst_abase + __ldg(A.dst.t + A.d_tb + lb);
  if (A.o0 >= 0) l.base += __ldg(A.dst.t + A.d_to0 + co0);
  if (A.o1 >= 0) l.base += __ldg(A.dst.t + A.d_to1 + co1);
  l.stride = A.dst_astride;
  if (A.dst_atab) l.tab = A.dst.t + A.d_ta;
  return l;
}

template <typename T, int KIND, bool AFAST, bool CHIRP>
struct Tile {
  using C = cplx<T>;
  static constexpr bool kReal = KIND == kR2C || KIND == kC2R;
  const StageArgs& A;
  const FlexArgs& F;
  C *s0, *s1;       // first / second exchange buffer
  int b0, nb;       // first line along b, lines (real lines of R2C / C2R) in the tile
  int nact;         // complex lines in the tile
  int co0, co1;

  // item it of cnt per line -> (line, j); false past the tile's lines
  __device__ __forceinline__ bool split(int it, int cnt, unsigned magic, int* line, int* j) const {
    if (AFAST) {
      *line = static_cast<int>(__umulhi(static_cast<unsigned>(it), magic));
      *j = it - *line * cnt;
    } else {
      *line = it & (F.B - 1);
      *j = it >> F.lshift;
    }
    return *line < nact;
  }
  // items of cnt per line a tile has (a-fast: of its present lines only)
  __device__ __forceinline__ int items(int cnt) const { return (AFAST ? nact : F.B) * cnt; }
  // element e of a line in an exchange buffer of pitch P
  __device__ __forceinline__ int at(int line, int e, int P) const { return AFAST ? line * P + e : e * F.B + line; }

  __device__ __forceinline__ C chirp(int k) const {
    return __ldg(reinterpret_cast<const C*>(F.chirp) + k);
  }

  // a thread's share of a line: positions k, k + step, ... of `line`
  __device__ __forceinline__ bool line_share(int* line, int* k, int* step) const {
    if (AFAST) {
      *step = F.share;
      *line = static_cast<int>(__umulhi(threadIdx.x, F.magic_share));
      *k = static_cast<int>(threadIdx.x) - *line * F.share;
    } else {
      *step = static_cast<int>(blockDim.x) >> F.lshift;
      *line = threadIdx.x & (F.B - 1);
      *k = static_cast<int>(threadIdx.x) >> F.lshift;
    }
    return *line < nact;
  }

  // value of an inverse C2C transform: real and imaginary parts swapped on the
  // way in and out of the forward codelets
  __device__ __forceinline__ C swapped(C c) const { return F.swap ? mk<T>(c.y, c.x) : c; }

  // C2R: the full spectrum Z = X0 + i X1 of a line pair from the two half
  // spectra (imaginary parts of DC and Nyquist dropped), parts swapped, into s1
  __device__ __forceinline__ void assemble() const {
    const int h = F.n / 2 + 1;
    int line, k, step;
    if (!line_share(&line, &k, &step)) return;
    const C* in = reinterpret_cast<const C*>(A.in);
    const C zero = mk<T>(T(0), T(0));
    const bool two = 2 * line + 1 < nb;
    const Line l0 = src_line(A, b0 + 2 * line, co0, co1);
    const Line l1 = two ? src_line(A, b0 + 2 * line + 1, co0, co1) : l0;
    for (; k < h; k += step) {
      const C x0 = in[l0.at(k)];
      const C x1 = two ? in[l1.at(k)] : zero;
      if (k == 0 || 2 * k == F.n) {
        s1[at(line, k, F.P1)] = mk<T>(x1.x, x0.x);
      } else {
        s1[at(line, k, F.P1)] = mk<T>(x0.y + x1.x, x0.x - x1.y);
        s1[at(line, F.n - k, F.P1)] = mk<T>(x1.x - x0.y, x0.x + x1.y);
      }
    }
  }

  // R2C: the two half spectra of a line pair from its full spectrum in z
  __device__ __forceinline__ void separate(const C* z, int P) const {
    const int h = F.n / 2 + 1;
    int line, k, step;
    if (!line_share(&line, &k, &step)) return;
    const T hs = T(0.5) * T(A.scale);
    C* out = reinterpret_cast<C*>(A.out);
    const bool two = 2 * line + 1 < nb;
    const Line l0 = dst_line(A, b0 + 2 * line, co0, co1);
    const Line l1 = two ? dst_line(A, b0 + 2 * line + 1, co0, co1) : l0;
    for (; k < h; k += step) {
      const C a = z[at(line, k, P)];
      const C b = cconj(z[at(line, k == 0 ? 0 : F.n - k, P)]);
      out[l0.at(k)] = cscale(cadd(a, b), hs);
      if (two) {
        const C d = csub(a, b);
        out[l1.at(k)] = mk<T>(d.y * hs, -d.x * hs);
      }
    }
  }

  // values of the R outputs v[r] at positions k0 + r * step of `line`, to the
  // destination (C2C, C2R) or to the line's natural order in z (R2C)
  template <int R>
  __device__ __forceinline__ void finish(C* v, int line, int k0, int step, C* z, int P) const {
    const int lim = F.n;
    if (CHIRP) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int k = k0 + r * step;
        if (k < lim) v[r] = cmul(v[r], chirp(k));
      }
    }
    if (KIND == kR2C) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int k = k0 + r * step;
        if (!CHIRP || k < lim) z[at(line, k, P)] = v[r];
      }
      return;
    }
    if (A.scale != 1.0) {
      const T s = T(A.scale);
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = cscale(v[r], s);
    }
    if (KIND == kC2R) {
      T* out = reinterpret_cast<T*>(A.out);
      const Line l0 = dst_line(A, b0 + 2 * line, co0, co1);
      each<R, CHIRP>(l0, k0, step, lim, [&](int r, int64_t o) { out[o] = v[r].y; });
      if (2 * line + 1 < nb) {
        const Line l1 = dst_line(A, b0 + 2 * line + 1, co0, co1);
        each<R, CHIRP>(l1, k0, step, lim, [&](int r, int64_t o) { out[o] = v[r].x; });
      }
    } else {
      C* out = reinterpret_cast<C*>(A.out);
      each<R, CHIRP>(dst_line(A, b0 + line, co0, co1), k0, step, lim,
                     [&](int r, int64_t o) { out[o] = swapped(v[r]); });
    }
  }

  // codelets over positions j + r R2 (r < R1); row j of the line's matrix
  template <int R>
  __device__ __forceinline__ void pass1() const {
    const int R2 = F.R2, lim = F.n;
    const C zero = mk<T>(T(0), T(0));
    for (int it = threadIdx.x; it < items(R2); it += blockDim.x) {
      int line, j;
      if (!split(it, R2, F.magic2, &line, &j)) continue;
      C v[R];
      if (KIND == kC2R) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int p = j + r * R2;
          v[r] = (!CHIRP || p < lim) ? s1[at(line, p, F.P1)] : zero;
        }
      } else if (KIND == kR2C) {
        const T* in = reinterpret_cast<const T*>(A.in);
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = zero;
        each<R, CHIRP>(src_line(A, b0 + 2 * line, co0, co1), j, R2, lim, [&](int r, int64_t o) { v[r].x = in[o]; });
        if (2 * line + 1 < nb)
          each<R, CHIRP>(src_line(A, b0 + 2 * line + 1, co0, co1), j, R2, lim,
                         [&](int r, int64_t o) { v[r].y = in[o]; });
      } else {
        const C* in = reinterpret_cast<const C*>(A.in);
        if (CHIRP) {
#pragma unroll
          for (int r = 0; r < R; ++r) v[r] = zero;
        }
        each<R, CHIRP>(src_line(A, b0 + line, co0, co1), j, R2, lim,
                       [&](int r, int64_t o) { v[r] = swapped(in[o]); });
      }
      if (CHIRP) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int p = j + r * R2;
          if (p < lim) v[r] = cmul(v[r], chirp(p));
        }
      }
      Dft<T, R>::run(v);
#pragma unroll
      for (int r = 0; r < R; ++r) s0[at(line, j * (AFAST ? (R | 1) : R) + r, F.P0)] = v[r];
    }
  }

  // columns of the R2 x R1 matrix: twiddles, codelets, outputs k = j + r R1.
  // Chirp-z: the filter, and the first pass of the inverse transform on the
  // same registers (its inputs are the positions j + r R1 too), row j of the
  // R1 x R2 matrix of the way back.
  template <int R>
  __device__ __forceinline__ void pass2() const {
    const int R1 = F.R1, R1p = AFAST ? (R1 | 1) : R1;
    const C* tw = reinterpret_cast<const C*>(F.tw);
    for (int it = threadIdx.x; it < items(R1); it += blockDim.x) {
      int line, j;
      if (!split(it, R1, F.magic1, &line, &j)) continue;
      C v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = s0[at(line, r * R1p + j, F.P0)];
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], __ldg(tw + r * R1 + j));
      Dft<T, R>::run(v);
      if (CHIRP) {
        const C* f = reinterpret_cast<const C*>(F.filter);
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = cmul(v[r], __ldg(f + j + r * R1));
        Dft<T, R>::run(v);  // inverse: output r is the forward output R - r
#pragma unroll
        for (int r = 0; r < R; ++r) s1[at(line, j * (AFAST ? (R | 1) : R) + r, F.P1)] = v[(R - r) % R];
      } else {
        finish<R>(v, line, j, R1, s1, F.P1);
      }
    }
  }

  // chirp-z: the second pass of the inverse transform, outputs k = j + r R2
  template <int R>
  __device__ __forceinline__ void pass3() const {
    const int R2 = F.R2, R2p = AFAST ? (R2 | 1) : R2;
    const C* tw = reinterpret_cast<const C*>(F.tw) + F.m;
    for (int it = threadIdx.x; it < items(R2); it += blockDim.x) {
      int line, j;
      if (!split(it, R2, F.magic2, &line, &j)) continue;
      C v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = s1[at(line, r * R2p + j, F.P1)];
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], cconj(__ldg(tw + r * R2 + j)));
      Dft<T, R>::run(v);
      C u[R];
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = v[(R - r) % R];
      finish<R>(u, line, j, R2, s0, F.P0);
    }
  }
};

// codelet lengths of the register classes (class 2: the partners that the most
// even split pairs a codelet above 16 with, 11 and 13 left out)
#define DFFT_FLEX_R0(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10)
#define DFFT_FLEX_R1(X) DFFT_FLEX_R0(X) X(11) X(12) X(13) X(14) X(15) X(16)
#define DFFT_FLEX_R2(X) \
  X(5) X(7) X(9) X(10) X(12) X(14) X(15) X(16) X(18) X(20) X(21) X(24) X(25) X(27) X(28) X(30) X(32)

template <int PASS, int CLS, typename TileT>
__device__ __forceinline__ void run_pass(const TileT& t, int R) {
#define DFFT_CASE(R_)                       \
  case R_:                                  \
    if constexpr (PASS == 1)                \
      t.template pass1<R_>();               \
    else if constexpr (PASS == 2)           \
      t.template pass2<R_>();               \
    else                                    \
      t.template pass3<R_>();               \
    break;
  if constexpr (CLS == 0) {
    switch (R) { DFFT_FLEX_R0(DFFT_CASE) default: break; }
  } else if constexpr (CLS == 1) {
    switch (R) { DFFT_FLEX_R1(DFFT_CASE) default: break; }
  } else {
    switch (R) { DFFT_FLEX_R2(DFFT_CASE) default: break; }
  }
#undef DFFT_CASE
}

template <typename T, int KIND, bool AFAST, int CLS, bool CHIRP>
__global__ void __launch_bounds__(Bounds<T, CLS>::threads, (Bounds<T, CLS>::blocks))
    fft_flex_kernel(const __grid_constant__ StageArgs A, const __grid_constant__ FlexArgs F) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using TileT = Tile<T, KIND, AFAST, CHIRP>;
  using C = cplx<T>;
  const int per = TileT::kReal ? 2 * F.B : F.B;
  const int b0 = static_cast<int>(blockIdx.x) * per, nb = min(per, A.Eb - b0);
  C* s0 = reinterpret_cast<C*>(smem_raw);
  const TileT t{A, F, s0, s0 + F.B * F.P0, b0, nb, TileT::kReal ? (nb + 1) / 2 : nb,
                static_cast<int>(blockIdx.y), static_cast<int>(blockIdx.z)};
  if (KIND == kC2R) {
    t.assemble();
    __syncthreads();
  }
  run_pass<1, CLS>(t, F.R1);
  __syncthreads();
  run_pass<2, CLS>(t, F.R2);
  if (CHIRP) {
    __syncthreads();
    run_pass<3, CLS>(t, F.R1);
  }
  if (KIND == kR2C) {
    __syncthreads();
    t.separate(CHIRP ? t.s0 : t.s1, CHIRP ? F.P0 : F.P1);
  }
}

template <typename T, int KIND, bool AFAST, int CLS, bool CHIRP>
cudaError_t launch_kernel(const StageArgs& A, const FlexArgs& F, cudaStream_t st) {
  auto k = fft_flex_kernel<T, KIND, AFAST, CLS, CHIRP>;
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k), F.smem);
  if (e != cudaSuccess) return e;
  k<<<fast_grid(A), F.nthreads, F.smem, st>>>(with_table_offsets(A), F);
  return cudaGetLastError();
}

// The kernels of one precision, register class and form: instantiated by
// fft_flex_inst.cu, one translation unit each.  Real lines are a-fast only.
template <typename T, int CLS, bool CHIRP>
cudaError_t launch_class(const StageArgs& A, const FlexArgs& F, int kind, cudaStream_t st);

}  // namespace flex
}  // namespace dev
}  // namespace dfft
