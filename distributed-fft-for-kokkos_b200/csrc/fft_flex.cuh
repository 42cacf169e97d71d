// Two-pass FFT stage for lines of m = R1 R2 points, R1 >= R2 two codelet
// lengths up to 32 (sm_100a): the 2^a 3^b 5^c 7^d lengths up to 512 that split
// so (and some up to 1024, and multiples of 11 and 13 up to 198), and, through
// the chirp-z convolution, every length n with a larger prime factor and
// 2 n - 1 <= 1024.
//
// What bounds it: bytes.  A tile of B lines is read from global memory once
// and written once; between the two passes a line crosses shared memory once
// (chirp-z: twice).  Pass 1 gives every thread one R1-point codelet whose
// inputs it loads itself, R1 independent loads in flight; it leaves row j of
// the line's R2 x R1 matrix in shared memory; pass 2 reads columns, applies
// the twiddle w_m^(j r) and stores straight to global memory.
//
// Measured (B200, forward + backward; before: the table-driven kernel of
// fft_stage.cu, five launches per chirp-z stage, the 24- and 8-value register
// kernels): 300 x 250 x 360 complex64 3818 -> 536 us, 200 x 180 x 252 R2C / C2R
// double 1633 -> 207 us, 131 x 105 x 157 R2C / C2R double 766 -> 190 us, 256^3
// complex128 644 -> 552 us, 384^3 R2C / C2R double 1568 -> 1124 us.  On 2^k and
// 3 2^k lines the tuner chooses between this kernel and the older ones, which
// stay ahead on complex64 (two lines per thread) and short stages.
//
// The radices are template arguments, a kernel per length: with run-time
// radices (a switch over codelets in one kernel: 810, 467, 331, 608 us and no
// gain above) the registers were those of the largest codelet and every
// shared-memory and global offset was computed, 90 instructions a point at
// 10-20 % occupancy.  Here offsets are immediates and the registers follow R1.
// CTAs are small (about 128 threads, one
// butterfly each per pass), so that an SM holds many, each at a different
// point between its loads and stores.
//
// Thread mapping: a-fast rows (unit stride along the FFT axis) take the
// butterflies of a line on consecutive threads, with the matrix rows padded
// to an odd pitch; b-fast rows (unit stride along the tile axis) take the B
// lines of a tile on consecutive threads, 128-byte rows.
//
// Inverse transforms take the forward codelets' outputs in reverse order,
// X_{m-k}.
//
// R2C / C2R lines go in pairs, one as the real and one as the imaginary part
// of a complex line, as in the other kernels.  Chirp-z ones go alone: a pair
// shares its rounding errors and its infinities, and the kernels that longer
// lines of these lengths take (bluestein.cu) do not pair.
#pragma once

#include "fft_codelet.cuh"

namespace dfft {
namespace dev {
namespace flex {

using codelet::Dft;

// Resident threads per SM the registers are sized for: what the R1 values of a
// thread, its addresses and the codelet's temporaries take with at most a few
// spills (more for the chirp-z form, `more`).  C2R lines, which load both half
// spectra, take a few more registers when left alone, and lose a CTA per SM by
// it (384^3 double: 221 us a launch at two CTAs of 210 registers, 186 at four).
template <typename T>
constexpr int resident_threads(int r, bool more, bool afast = false) {
  if (sizeof(T) == 4)
    return more ? (r <= 12 ? 896 : r <= 16 ? 768 : r <= 21 ? 576 : 512)
                : (r <= 8 ? 1280 : r <= 12 ? 1024 : r <= 16 ? 896 : r <= 21 ? 640 : r <= 25 ? 576 : 512);
  return more ? (r <= 8 ? 768 : r <= 10 ? 640 : r <= 16 ? 512 : r <= 21 ? 384 : r <= 25 ? 320 : 256)
              : (r <= 8 ? 896 : r <= 10 ? 768 : r <= 12 ? 640 : r <= 16 ? 512 : r <= 21 ? 448
                 : r <= 24 && afast ? 512 : r <= 25 ? 384 : 256);
}

// Lines per tile: about 128 threads.  b-fast rows of 128 bytes; of 64 bytes for
// complex64 lines with R1 >= 12, whose 128-byte tiles are CTAs of 200 to 400
// threads that spend their time at the barrier (300 x 250 x 360: stages of 104
// and 103 us with 16 lines, 97 and 86 us with 8).
template <typename T>
constexpr int tile_lines(bool afast, int r) {
  if (afast) return 128 / r > 1 ? 128 / r : 1;
  int b = sizeof(T) == 4 && r < 12 ? 16 : 8;
  while (b * r < 64) b *= 2;
  return b;
}

template <typename T, int KIND, bool AFAST, int R1, int R2, bool CHIRP>
struct Shape {
  static constexpr int B = tile_lines<T>(AFAST, R1);
  static constexpr int NT = (B * R1 + 31) / 32 * 32;
  // a line's elements in shared memory: the R2 x R1 matrix (chirp-z: also the
  // R1 x R2 one of the way back), or the line in natural order
  static constexpr int m = R1 * R2, odd1 = R1 | 1, odd2 = R2 | 1;
  static constexpr int p1 = R2 * odd1, p2 = CHIRP ? R1 * odd2 : 0, pn = m | 1;
  static constexpr int P = AFAST ? (p1 > p2 ? (p1 > pn ? p1 : pn) : (p2 > pn ? p2 : pn)) : m;
  static constexpr size_t smem = sizeof(cplx<T>) * B * P;
  static constexpr int fit = resident_threads<T>(R1, CHIRP, AFAST) / NT;
  static constexpr int blocks = fit > 0 ? fit : 1;
};

// positions of a line: affine, or from the axis table
struct Line {
  int64_t base;
  int stride;
  const int64_t* tab;
};

__device__ __forceinline__ Line src_line(const StageArgs& A, int lb, int co0, int co1) {
  Line l;
  l.tab = nullptr;
  if (A.src_line_affine) {
    int64_t s;
    radix::line_affine(A.src, A, lb, co0, co1, &l.base, &s);
    l.stride = static_cast<int>(s);
    return l;
  }
  l.base = A.src_abase + __ldg(A.src.t + A.s_tb + lb);
  if (A.o0 >= 0) l.base += __ldg(A.src.t + A.s_to0 + co0);
  if (A.o1 >= 0) l.base += __ldg(A.src.t + A.s_to1 + co1);
  l.stride = static_cast<int>(A.src_astride);
  if (A.src_atab) l.tab = A.src.t + A.s_ta;
  return l;
}

__device__ __forceinline__ Line dst_line(const StageArgs& A, int lb, int co0, int co1) {
  Line l;
  l.tab = nullptr;
  if (A.dst_line_affine) {
    int64_t s;
    radix::line_affine(A.dst, A, lb, co0, co1, &l.base, &s);
    l.stride = static_cast<int>(s);
    return l;
  }
  l.base = A.dst_abase + __ldg(A.dst.t + A.d_tb + lb);
  if (A.o0 >= 0) l.base += __ldg(A.dst.t + A.d_to0 + co0);
  if (A.o1 >= 0) l.base += __ldg(A.dst.t + A.d_to1 + co1);
  l.stride = static_cast<int>(A.dst_astride);
  if (A.dst_atab) l.tab = A.dst.t + A.d_ta;
  return l;
}

// f(r, offset of position p0 + r * STEP of the line) for r < R; LIM: only
// positions below lim.  a-fast lines have unit stride.
template <int R, int STEP, bool AFAST, bool LIM, typename Fn>
__device__ __forceinline__ void positions(const Line& l, int p0, int lim, Fn&& f) {
  if (l.tab) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (!LIM || p0 + r * STEP < lim) f(r, l.base + __ldg(l.tab + p0 + r * STEP));
  } else if (AFAST) {
    const int64_t b = l.base + p0;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (!LIM || p0 + r * STEP < lim) f(r, b + r * STEP);
  } else {
    // (len - 1) * stride < 2^31 (host check)
    const int64_t b = l.base + static_cast<int64_t>(p0) * l.stride;
    const int st = STEP * l.stride;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (!LIM || p0 + r * STEP < lim) f(r, b + r * st);
  }
}

// The same for outputs k = j + r * STEP of an m-point transform, m - k for
// inverse ones (position 0 stays).
template <int R, int STEP, int M, bool AFAST, typename Fn>
__device__ __forceinline__ void outputs(const Line& l, int j, bool inverse, Fn&& f) {
  if (!inverse) {
    positions<R, STEP, AFAST, false>(l, j, 0, f);
    return;
  }
  const int p0 = j == 0 ? 0 : M - j;
  if (l.tab) {
    f(0, l.base + __ldg(l.tab + p0));
#pragma unroll
    for (int r = 1; r < R; ++r) f(r, l.base + __ldg(l.tab + M - j - r * STEP));
  } else if (AFAST) {
    f(0, l.base + p0);
    const int64_t b = l.base + M - j;
#pragma unroll
    for (int r = 1; r < R; ++r) f(r, b - r * STEP);
  } else {
    f(0, l.base + static_cast<int64_t>(p0) * l.stride);
    const int64_t b = l.base + static_cast<int64_t>(M - j) * l.stride;
    const int st = STEP * l.stride;
#pragma unroll
    for (int r = 1; r < R; ++r) f(r, b - r * st);
  }
}

// Column j of the matrix of R1 wide rows: R values, twiddled (tw [r][j] = w^(j r)).
template <typename T, int R, int R1, int PITCH>
__device__ __forceinline__ void load_column(const cplx<T>* s, const cplx<T>* tw, int j, cplx<T>* v) {
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = s[r * PITCH];
#pragma unroll
  for (int r = 1; r < R; ++r) v[r] = cmul(v[r], __ldg(tw + r * R1 + j));
}

template <typename T, int KIND, bool AFAST, int R1, int R2, bool CHIRP>
__global__ void __launch_bounds__((Shape<T, KIND, AFAST, R1, R2, CHIRP>::NT),
                                  (Shape<T, KIND, AFAST, R1, R2, CHIRP>::blocks))
    fft_flex_kernel(const __grid_constant__ StageArgs A, const __grid_constant__ FlexArgs F) {
  using C = cplx<T>;
  using S = Shape<T, KIND, AFAST, R1, R2, CHIRP>;
  constexpr bool kPairs = (KIND == kR2C || KIND == kC2R) && !CHIRP;  // two real lines a complex line
  constexpr int B = S::B, M = S::m;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const s = reinterpret_cast<C*>(smem_raw);
  release_dependents();
  const int t = threadIdx.x;
  const int per = kPairs ? 2 * B : B;
  const int b0 = static_cast<int>(blockIdx.x) * per, nb = min(per, A.Eb - b0);
  const int nact = kPairs ? (nb + 1) / 2 : nb;  // complex lines in the tile
  const int co0 = blockIdx.y, co1 = blockIdx.z;
  const int n = CHIRP ? F.n : M;
  const bool inverse = KIND == kC2R || F.inverse;
  // chirp-z of the inverse: the conjugate chirp and the filter made from it
  auto chirp = [&](int k) {
    C c = __ldg(reinterpret_cast<const C*>(F.chirp) + k);
    if (inverse) c.y = -c.y;
    return c;
  };
  // element e of a line
  auto at = [&](int line, int e) -> C& { return AFAST ? s[line * S::P + e] : s[e * B + line]; };
  constexpr int row1 = AFAST ? S::odd1 : R1, row2 = AFAST ? S::odd2 : R2;  // matrix row pitch
  constexpr int el = AFAST ? 1 : B;                                        // pitch of neighbouring elements

  // thread -> (line, j) among cnt butterflies a line
  const int line2 = AFAST ? t / R2 : t % B, j2 = AFAST ? t % R2 : t / B;
  const int line1 = AFAST ? t / R1 : t % B, j1 = AFAST ? t % R1 : t / B;
  const bool act2 = (AFAST ? t < B * R2 : j2 < R2) && line2 < nact;
  const bool act1 = (AFAST ? t < B * R1 : j1 < R1) && line1 < nact;

  dependency_wait();
  // ---- pass 1: codelets over positions j + r R2, row j of the matrix
  C v[R1];
  if (act2) {
    if constexpr (CHIRP) {
#pragma unroll
      for (int r = 0; r < R1; ++r) v[r] = mk<T>(T(0), T(0));
      const Line l = src_line(A, b0 + line2, co0, co1);
      if constexpr (KIND == kR2C) {
        const T* in = reinterpret_cast<const T*>(A.in);
        positions<R1, R2, AFAST, true>(l, j2, n, [&](int r, int64_t o) { v[r].x = in[o]; });
      } else if constexpr (KIND == kC2R) {
        // the full line from its half spectrum (imaginary parts of DC and
        // Nyquist dropped), every mode loaded for both positions it makes
        const C* x = reinterpret_cast<const C*>(A.in) + l.base;
        const T wt = T(A.weight);
#pragma unroll
        for (int r = 0; r < R1; ++r) {
          const int p = j2 + r * R2;
          if (p >= n) continue;
          const int q = 2 * p > n ? n - p : p;
          const C c = x[q];
          v[r] = (q == 0 || 2 * q == n) ? mk<T>(c.x, T(0)) : mk<T>(c.x * wt, (q < p ? -c.y : c.y) * wt);
        }
      } else {
        const C* in = reinterpret_cast<const C*>(A.in);
        positions<R1, R2, AFAST, true>(l, j2, n, [&](int r, int64_t o) { v[r] = in[o]; });
      }
#pragma unroll
      for (int r = 0; r < R1; ++r)
        if (j2 + r * R2 < n) v[r] = cmul(v[r], chirp(j2 + r * R2));
    } else if constexpr (KIND == kR2C) {
      const T* in = reinterpret_cast<const T*>(A.in);
#pragma unroll
      for (int r = 0; r < R1; ++r) v[r] = mk<T>(T(0), T(0));
      positions<R1, R2, AFAST, false>(src_line(A, b0 + 2 * line2, co0, co1), j2, 0,
                                      [&](int r, int64_t o) { v[r].x = in[o]; });
      if (2 * line2 + 1 < nb)
        positions<R1, R2, AFAST, false>(src_line(A, b0 + 2 * line2 + 1, co0, co1), j2, 0,
                                        [&](int r, int64_t o) { v[r].y = in[o]; });
    } else if constexpr (KIND == kC2R) {
      // Z from the half spectra directly, every mode loaded for both positions
      // it makes: assembled in shared memory, with the barriers that takes,
      // 384^3 double took 273 us where this form took 221
      const bool two = 2 * line2 + 1 < nb;
      const C* x0 = reinterpret_cast<const C*>(A.in) + src_line(A, b0 + 2 * line2, co0, co1).base;
      const C* x1 = two ? reinterpret_cast<const C*>(A.in) + src_line(A, b0 + 2 * line2 + 1, co0, co1).base : x0;
      const T wt = T(A.weight);
#pragma unroll
      for (int r = 0; r < R1; ++r) {
        const int p = j2 + r * R2;
        const bool mirror = 2 * p > M;
        const int q = mirror ? M - p : p;
        C c0 = x0[q];
        C c1 = two ? x1[q] : mk<T>(T(0), T(0));
        if (q == 0 || 2 * q == M) {
          v[r] = mk<T>(c0.x, c1.x);
        } else {
          c0 = cscale(c0, wt);
          c1 = cscale(c1, wt);
          v[r] = mirror ? mk<T>(c0.x + c1.y, c1.x - c0.y) : mk<T>(c0.x - c1.y, c0.y + c1.x);
        }
      }
    } else {
      const C* in = reinterpret_cast<const C*>(A.in);
      positions<R1, R2, AFAST, false>(src_line(A, b0 + line2, co0, co1), j2, 0,
                                      [&](int r, int64_t o) { v[r] = in[o]; });
    }
    Dft<T, R1>::run(v);
    C* o = &at(line2, j2 * row1);
#pragma unroll
    for (int r = 0; r < R1; ++r) o[r * el] = v[r];
  }
  __syncthreads();

  const C* tw = reinterpret_cast<const C*>(F.tw);
  const T scale = T(A.scale);
  if constexpr (!CHIRP) {
    // ---- pass 2: columns, outputs k = j + r R1
    C u[R2];
    if (act1) {
      load_column<T, R2, R1, row1 * el>(&at(line1, j1), tw, j1, u);
      Dft<T, R2>::run(u);
    }
    if constexpr (KIND == kC2C) {
      if (act1) {
        if (A.scale != 1.0) {
#pragma unroll
          for (int r = 0; r < R2; ++r) u[r] = cscale(u[r], scale);
        }
        C* out = reinterpret_cast<C*>(A.out);
        outputs<R2, R1, M, AFAST>(dst_line(A, b0 + line1, co0, co1), j1, inverse,
                                  [&](int r, int64_t o) { out[o] = u[r]; });
      }
      return;
    }
    if constexpr (KIND == kC2R) {
      if (act1) {
        T* out = reinterpret_cast<T*>(A.out);
        outputs<R2, R1, M, AFAST>(dst_line(A, b0 + 2 * line1, co0, co1), j1, true,
                                  [&](int r, int64_t o) { out[o] = u[r].x * scale; });
        if (2 * line1 + 1 < nb)
          outputs<R2, R1, M, AFAST>(dst_line(A, b0 + 2 * line1 + 1, co0, co1), j1, true,
                                    [&](int r, int64_t o) { out[o] = u[r].y * scale; });
      }
      return;
    }
    __syncthreads();  // every column read: the buffer takes the line in natural order
    if (act1) {
#pragma unroll
      for (int r = 0; r < R2; ++r) at(line1, j1 + r * R1) = u[r];
    }
  } else {
    // ---- pass 2: columns, the filter, and the first pass of the inverse
    // transform on the same registers (its inputs are the positions j + r R1
    // too): row j of the R1 x R2 matrix of the way back
    C u[R2];
    if (act1) {
      load_column<T, R2, R1, row1 * el>(&at(line1, j1), tw, j1, u);
      Dft<T, R2>::run(u);
      const C* f = reinterpret_cast<const C*>(inverse ? F.filter_inverse : F.filter);
#pragma unroll
      for (int r = 0; r < R2; ++r) u[r] = cmul(u[r], __ldg(f + j1 + r * R1));
      Dft<T, R2>::run(u);  // inverse: output r is the forward output R2 - r
    }
    __syncthreads();
    if (act1) {
      C* o = &at(line1, j1 * row2);
#pragma unroll
      for (int r = 0; r < R2; ++r) o[r * el] = u[(R2 - r) % R2];
    }
    __syncthreads();
    // ---- pass 3: outputs k = j + r R2
    C w[R1];
    if (act2) {
      const C* c = &at(line2, j2);
#pragma unroll
      for (int r = 0; r < R1; ++r) w[r] = c[r * row2 * el];
#pragma unroll
      for (int r = 1; r < R1; ++r) w[r] = cmul(w[r], cconj(__ldg(tw + M + r * R2 + j2)));
      Dft<T, R1>::run(w);
      C x[R1];
#pragma unroll
      for (int r = 0; r < R1; ++r) {
        x[r] = w[(R1 - r) % R1];
        if (j2 + r * R2 < n) x[r] = cmul(x[r], chirp(j2 + r * R2));
      }
      const Line l = dst_line(A, b0 + line2, co0, co1);
      if constexpr (KIND == kC2C) {
        C* out = reinterpret_cast<C*>(A.out);
        positions<R1, R2, AFAST, true>(l, j2, n, [&](int r, int64_t o) { out[o] = cscale(x[r], scale); });
      } else if constexpr (KIND == kC2R) {
        T* out = reinterpret_cast<T*>(A.out);
        positions<R1, R2, AFAST, true>(l, j2, n, [&](int r, int64_t o) { out[o] = x[r].x * scale; });
      } else {
        C* out = reinterpret_cast<C*>(A.out);
        const T sw = scale * T(A.weight);
        positions<R1, R2, AFAST, true>(l, j2, n / 2 + 1, [&](int r, int64_t o) {
          const int k = j2 + r * R2;
          out[o] = (k == 0 || 2 * k == n) ? mk<T>(x[r].x * scale, T(0)) : cscale(x[r], sw);
        });
      }
    }
    return;
  }
  // ---- R2C: the two half spectra of a line pair from its full spectrum
  if constexpr (KIND == kR2C && !CHIRP) {
    __syncthreads();
    constexpr int TPL = S::NT / B;  // threads a line
    const int line = t / TPL;
    if (line < nact) {
      C* out = reinterpret_cast<C*>(A.out);
      const T h0 = T(0.5) * scale, h1 = h0 * T(A.weight);
      const bool two = 2 * line + 1 < nb;
      C* y0 = out + dst_line(A, b0 + 2 * line, co0, co1).base;
      C* y1 = two ? out + dst_line(A, b0 + 2 * line + 1, co0, co1).base : y0;
      for (int k = t % TPL; k <= M / 2; k += TPL) {
        const C a = at(line, k);
        const C b = cconj(at(line, k == 0 ? 0 : M - k));
        const T hs = (k == 0 || 2 * k == M) ? h0 : h1;
        y0[k] = cscale(cadd(a, b), hs);
        if (two) {
          const C d = csub(a, b);
          y1[k] = mk<T>(d.y * hs, -d.x * hs);
        }
      }
    }
  }
}

using LaunchFn = cudaError_t (*)(const StageArgs& A, const FlexArgs& F, cudaStream_t st);

template <typename T, int KIND, bool AFAST, int R1, int R2, bool CHIRP>
cudaError_t launch_kernel(const StageArgs& A, const FlexArgs& F, cudaStream_t st) {
  using S = Shape<T, KIND, AFAST, R1, R2, CHIRP>;
  auto k = fft_flex_kernel<T, KIND, AFAST, R1, R2, CHIRP>;
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k), S::smem);
  if (e != cudaSuccess) return e;
  return launch_kernel_early(early_start(A, sizeof(cplx<T>)), k, fast_grid(A), S::NT, S::smem, st, with_table_offsets(A), F);
}

// The kernels of one length: C2C a-fast and b-fast, R2C and C2R (a-fast).
struct Entry {
  int m;
  LaunchFn c2c_a, c2c_b, r2c, c2r;
};
// The entries of one group of lengths (fft_flex_lengths.h), defined by
// fft_flex_inst.cu in a translation unit each.
template <typename T, bool CHIRP, int GROUP>
struct Group {
  static const Entry* entries(int* count);
};

}  // namespace flex
}  // namespace dev
}  // namespace dfft
