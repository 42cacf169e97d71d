// Line kernels of the Navier-Stokes right-hand side on its own arrays
// (sm_100a): transforms along x, y and z with the spectral operators, the
// advection product and the Runge-Kutta update folded into their loads and
// stores.
//
// What bounds the right-hand side: bytes.  Four backward and one forward
// transform of three components as separate stages move every spectrum and
// every physical field through memory at each of them.  Three facts make most
// of that unnecessary:
//   * the 2/3 rule keeps kx x ky x kz modes, about 8/27 of the spectrum, and a
//     line along y or z whose fixed modes are cut is zero, so the arrays hold
//     kept modes only: (x, y, z) kept before the x transforms, (y, z) kept
//     between x and y, z kept between y and z;
//   * i k_y and i k_z commute with the transforms along the other axes, so the
//     x transforms run on u and i k_x u only, the y transforms on u, i k_y u
//     and i k_x u, and only the z transforms on all four;
//   * the physical velocity and its gradient of a grid line are needed by the
//     advection product of that line alone, so the z kernel transforms the 12
//     fields of a pair of lines back, forms u . grad u and transforms its 3
//     components forward in shared memory: no physical field is written.
// The adjoint runs the transposes of the same steps.
// Measured (B200; before: four backward transforms and one forward of the plan
// around pointwise kernels): physical field to physical field over one RK4
// step, 192^3 FP32 4172 -> 1579 us; step and gradient, 96^3 FP64 4771 -> 1216 us.
//
// Each kernel is two passes of register codelets around one exchange, a kernel
// per length (as in fft_flex.cuh).  Inverse transforms take the forward
// codelets' outputs in reverse order.
#pragma once

#include "fft_flex.cuh"

namespace dfft {
namespace dev {
namespace nsl {

using codelet::Dft;

// one axis: n points, its kept modes -c .. c (x, y: k = 2 c + 1) or 0 .. c (z:
// k = c + 1), twiddles [r < R2][j < R1] of n = R1 R2
struct Axis {
  int n, c, k;
  const void* tw;
};

struct Grid {
  Axis x, y, z;
  double kscale;       // wavenumber = mode * kscale
  unsigned magic_kz;   // ceil(2^32 / z.k)
};

// kept index of position p of a full axis, -1 if cut; mode of a kept index
__device__ __forceinline__ int kept(const Axis& a, int p) {
  return p <= a.c ? p : (p >= a.n - a.c ? p - a.n + a.k : -1);
}
__device__ __forceinline__ int mode(const Axis& a, int i) { return i <= a.c ? i : i - a.k; }

template <typename T>
__device__ __forceinline__ cplx<T> ik(T k, cplx<T> v) {  // i k v
  return mk<T>(-k * v.y, k * v.x);
}

// q = first * kz + second
__device__ __forceinline__ void split_kz(const Grid& g, int q, int* first, int* second) {
  *first = g.z.k == 1 ? q : static_cast<int>(__umulhi(static_cast<unsigned>(q), g.magic_kz));
  *second = q - *first * g.z.k;
}

// Lines along x or y: B neighbouring lines a CTA, one component (blockIdx.y)
// and field (blockIdx.z).  Arrays in C order, Q = ky kz:
//   XInverse  (3, kx, Q) -> (nf, 3, nx, Q): field 1 is i k_x times field 0
//   YInverse  (2 or 1, 3, nx, ky, kz) -> (nf, 3, nx, ny, kz): fields U, i k_y U
//             and V of the fields U, V of XInverse
//   YForward  (nf, 3, nx, ny, kz) -> (nf, 3, nx, ky, kz)
//   XForward  (nf, 3, nx, Q) -> (nf, 3, kx, Q); adjoint: fields W, Hy, Hx in,
//             W - i k_y Hy and Hx out
enum LineKind { kXInverse, kYInverse, kYForward, kXForward };

template <typename T>
struct LineArgs {
  Grid g;
  const cplx<T>* in;
  cplx<T>* out;
  int lines;
  int adjoint;
};

template <typename T, int R1, int R2>
struct LineShape {
  static constexpr int B = flex::tile_lines<T>(false, R1);
  static constexpr size_t smem = sizeof(cplx<T>) * B * R1 * R2;
  static constexpr int NT = (B * R1 + 31) / 32 * 32;
  static constexpr int fit = (sizeof(T) == 4 && R1 <= 16 ? 896 : flex::resident_threads<T>(R1, true)) / NT;
  static constexpr int blocks = fit > 0 ? fit : 1;
};

template <typename T, int KIND, int R1, int R2>
__global__ void __launch_bounds__((LineShape<T, R1, R2>::NT), (LineShape<T, R1, R2>::blocks))
    ns_line_kernel(const __grid_constant__ LineArgs<T> a) {
  using C = cplx<T>;
  constexpr int B = LineShape<T, R1, R2>::B, N = R1 * R2;
  constexpr bool kX = KIND == kXInverse || KIND == kXForward;
  constexpr bool kInverse = KIND == kXInverse || KIND == kYInverse;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const s = reinterpret_cast<C*>(smem_raw);
  release_dependents();
  const Axis& ax = kX ? a.g.x : a.g.y;
  const int line = threadIdx.x % B, j = threadIdx.x / B;
  const int q = static_cast<int>(blockIdx.x) * B + line, d = blockIdx.y, f = blockIdx.z;
  const bool live = q < a.lines;
  const int kz = a.g.z.k;
  // a line's first element and the step along it, on the side of the points
  // (n positions) and of the modes (k kept ones); f0: source field
  const int f0 = KIND == kYInverse ? (f == 2 ? 1 : 0) : (KIND == kXForward && a.adjoint && f == 1) ? 2
                                                     : KIND == kXInverse ? 0 : f;
  int step;
  int64_t points, modes;
  int first = 0, second = 0;  // q = (y mode, z) or (x, z)
  split_kz(a.g, live ? q : 0, &first, &second);
  const int fp = kInverse ? f : f0, fm = kInverse ? f0 : f;  // fields of the two sides
  if (kX) {
    step = a.lines;
    points = static_cast<int64_t>(fp * 3 + d) * ax.n * step + q;
    modes = static_cast<int64_t>(fm * 3 + d) * ax.k * step + q;
  } else {
    step = kz;
    points = (static_cast<int64_t>(fp * 3 + d) * a.g.x.n + first) * ax.n * kz + second;
    modes = (static_cast<int64_t>(fm * 3 + d) * a.g.x.n + first) * ax.k * kz + second;
  }
  dependency_wait();
  if (live && j < R2) {
    C v[R1];
    if (kInverse) {
      const C* p = a.in + modes;
#pragma unroll
      for (int r = 0; r < R1; ++r) {
        const int i = kept(ax, j + r * R2);
        v[r] = i >= 0 ? p[i * step] : mk<T>(T(0), T(0));
      }
      if (f == 1) {
#pragma unroll
        for (int r = 0; r < R1; ++r) {
          const int p0 = j + r * R2;
          v[r] = ik<T>(T((2 * p0 < N ? p0 : p0 - N) * a.g.kscale), v[r]);  // cut modes are zero
        }
      }
    } else {
      const C* p = a.in + points + static_cast<int64_t>(j) * step;
#pragma unroll
      for (int r = 0; r < R1; ++r) v[r] = p[r * R2 * step];
      if (KIND == kXForward && a.adjoint && f == 0) {
        const C* h = p + static_cast<int64_t>(3) * ax.n * step;
        const T k = T(-mode(a.g.y, first) * a.g.kscale);
#pragma unroll
        for (int r = 0; r < R1; ++r) v[r] = cadd(v[r], ik<T>(k, h[r * R2 * step]));
      }
    }
    Dft<T, R1>::run(v);
    C* o = s + j * R1 * B + line;
#pragma unroll
    for (int r = 0; r < R1; ++r) o[r * B] = v[r];
  }
  __syncthreads();
  if (live && j < R1) {
    C u[R2];
    flex::load_column<T, R2, R1, R1 * B>(s + j * B + line, reinterpret_cast<const C*>(ax.tw), j, u);
    Dft<T, R2>::run(u);
    if (kInverse) {
      C* p = a.out + points;
      p[static_cast<int64_t>(j == 0 ? 0 : N - j) * step] = u[0];
      p += static_cast<int64_t>(N - j) * step;
#pragma unroll
      for (int r = 1; r < R2; ++r) p[-(r * R1 * step)] = u[r];
    } else {
      C* p = a.out + modes;
#pragma unroll
      for (int r = 0; r < R2; ++r) {
        const int i = kept(ax, j + r * R1);
        if (i >= 0) p[i * step] = u[r];
      }
    }
  }
}

// ---- along z: a pair of grid lines (x, y) and its neighbour, every real line
// pair one complex line (part x: the first point, part y: the second).
// Forward form: fields A, B, C of (u, i k_y u, i k_x u) and D = i k_z A back,
// u . grad u, 3 lines forward, written over field A.
// Adjoint form: also lambda (weight 1/2 on the interior modes times lscale)
// back; lambda_u = sum_j lambda_j d_a u_j and h_a,j = u_a lambda_j forward
// (weight 2 on the interior modes); W = lambda_u^ - i k_z h_z^ over field A,
// h_y^ over B, h_x^ over C.
// Every spectrum element is read once, scaled, and put to both positions of its
// line that it makes; codelets that loaded their positions themselves read
// each element twice with index and sign choices per position (192^3 FP32: 221
// us a launch, 154 us this way, 148 with four
// elements of a thread in flight).
template <typename T>
struct ZArgs {
  Grid g;
  cplx<T>* f;             // (3, 3, nx ny, kz)
  const cplx<T>* lambda;  // adjoint: (3, nx ny, kz)
  int points;             // nx ny
  double back, fwd, lscale;  // scale of the backward / forward transforms, of lambda
};

template <typename T, int R1, int R2, bool ADJ>
struct ZShape {
  static constexpr int back = ADJ ? 15 : 12;  // lines of a pair transformed to points
  static constexpr int fwd = ADJ ? 12 : 3;    // and to modes
  static constexpr int N = R1 * R2, odd1 = R1 | 1;
  static constexpr int P = R2 * odd1 > (N | 1) ? R2 * odd1 : (N | 1);  // pitch of a line
  // point pairs a CTA: about 192 butterflies; threads: one butterfly each, at most 256
  static constexpr int G = 192 / (back * R1) > 1 ? 192 / (back * R1) : 1;
  static constexpr int items = (G * back * R1 + 31) / 32 * 32;
  static constexpr int NT = items <= 256 ? items : (items / 2 + 31) / 32 * 32 <= 256 ? (items / 2 + 31) / 32 * 32 : 256;
  static constexpr size_t smem = 2 * sizeof(cplx<T>) * G * back * P;
  static constexpr bool ok = smem <= 227 * 1024;
  static constexpr int fit = (sizeof(T) == 4 && R1 <= 16 ? 960 : flex::resident_threads<T>(R1, true)) / NT;
  static constexpr int blocks = fit > 0 ? fit : 1;
};

template <typename T>
__device__ __forceinline__ cplx<T> mul2(cplx<T> a, cplx<T> b) {  // part by part: two grid points
  return mk<T>(a.x * b.x, a.y * b.y);
}

template <typename T, int R1, int R2, bool ADJ>
__global__ void __launch_bounds__((ZShape<T, R1, R2, ADJ>::NT), (ZShape<T, R1, R2, ADJ>::blocks))
    ns_z_kernel(const __grid_constant__ ZArgs<T> a) {
  using C = cplx<T>;
  using S = ZShape<T, R1, R2, ADJ>;
  constexpr int NB = S::back, NF = S::fwd, N = S::N, P = S::P, NT = S::NT, row = S::odd1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  release_dependents();
  C* const s0 = reinterpret_cast<C*>(smem_raw);
  C* const s1 = s0 + S::G * NB * P;
  const Axis& z = a.g.z;
  const C* tw = reinterpret_cast<const C*>(z.tw);
  const int c = z.c, kz = z.k;
  const int pair0 = static_cast<int>(blockIdx.x) * S::G;
  const int npair = min(S::G, (a.points + 1) / 2 - pair0);
  const C zero = mk<T>(T(0), T(0));
  dependency_wait();

  // assemble: Z = X0 + i X1 of every line from the kept modes of the two
  // points, scaled, in natural order (the cut positions are not written);
  // line = pair * NB + field * 3 + component, field 0 A, 1 B, 2 C, 3 D = i k_z A,
  // 4 lambda
  constexpr int NI = ADJ ? 12 : 9;  // lines read: A, B, C (and lambda)
  constexpr int U = 4;              // items a thread has in flight
  const int items = npair * NI * kz;
  for (int it0 = threadIdx.x; it0 < items; it0 += U * NT) {
    C c0[U], c1[U];
    int line[U], mode[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int it = min(it0 + u * NT, items - 1);  // (past the end: a load of the last item, not put)
      int ln;
      split_kz(a.g, it, &ln, &mode[u]);
      const int pr = ln / NI, l = ln % NI;
      const int64_t pt = 2 * static_cast<int64_t>(pair0 + pr);
      const C* x0 = (ADJ && l >= 9 ? a.lambda + static_cast<int64_t>(l - 9) * a.points * kz
                                   : a.f + static_cast<int64_t>(l) * a.points * kz) + pt * kz + mode[u];
      line[u] = pr * NB + l;
      c0[u] = x0[0];
      c1[u] = pt + 1 < a.points ? x0[kz] : zero;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (it0 + u * NT >= items) break;
      const int m = mode[u], l = line[u] % NB;
      const T sc = ADJ && l >= 9 ? T((m == 0 ? 1.0 : 0.5) * a.lscale) : T(a.back);
      auto put = [&](int ln, C p, C q) {
        C* o = s1 + ln * P;
        if (m == 0) {  // the imaginary part of the zero mode dropped
          o[0] = mk<T>(p.x, q.x);
        } else {
          o[m] = mk<T>(p.x - q.y, p.y + q.x);
          o[N - m] = mk<T>(p.x + q.y, q.x - p.y);
        }
      };
      const C p = cscale(c0[u], sc), q = cscale(c1[u], sc);
      put(ADJ && l >= 9 ? line[u] + 3 : line[u], p, q);
      if (l < 3) {
        const T k = T(m * a.g.kscale);
        put(line[u] + 9, ik<T>(k, p), ik<T>(k, q));
      }
    }
  }
  __syncthreads();
  // back, pass 1
  for (int it = threadIdx.x; it < npair * NB * R2; it += NT) {
    const int line = it / R2, j = it % R2;
    const C* b = s1 + line * P + j;
    C v[R1];
#pragma unroll
    for (int r = 0; r < R1; ++r) {
      const int p = j + r * R2;
      v[r] = static_cast<unsigned>(p - c - 1) < static_cast<unsigned>(N - 2 * c - 1) ? zero : b[r * R2];
    }
    Dft<T, R1>::run(v);
    C* o = s0 + line * P + j * row;
#pragma unroll
    for (int r = 0; r < R1; ++r) o[r] = v[r];
  }
  __syncthreads();
  // back, pass 2: points in natural order
  for (int it = threadIdx.x; it < npair * NB * R1; it += NT) {
    const int line = it / R1, j = it % R1;
    C u[R2];
    flex::load_column<T, R2, R1, row>(s0 + line * P + j, tw, j, u);
    Dft<T, R2>::run(u);
    C* o = s1 + line * P;
    o[j == 0 ? 0 : N - j] = u[0];
    o += N - j;
#pragma unroll
    for (int r = 1; r < R2; ++r) o[-r * R1] = u[r];
  }
  __syncthreads();
  // products at the points: s1 (12 or 15 lines a pair) -> s0 (3 or 12 lines)
  for (int it = threadIdx.x; it < npair * N; it += NT) {
    const int pr = it / N, i = it % N;
    const C* b = s1 + pr * NB * P + i;
    C* o = s0 + pr * NF * P + i;
    C u[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) u[d] = b[d * P];
    constexpr int grad[3] = {6, 3, 9};  // lines of d/dx, d/dy, d/dz
    if constexpr (!ADJ) {
#pragma unroll
      for (int d = 0; d < 3; ++d)
        o[d * P] = cadd(cadd(mul2<T>(u[0], b[(6 + d) * P]), mul2<T>(u[1], b[(3 + d) * P])), mul2<T>(u[2], b[(9 + d) * P]));
    } else {
      C la[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) la[d] = b[(12 + d) * P];
#pragma unroll
      for (int x = 0; x < 3; ++x)
        o[x * P] = cadd(cadd(mul2<T>(la[0], b[(grad[x] + 0) * P]), mul2<T>(la[1], b[(grad[x] + 1) * P])),
                        mul2<T>(la[2], b[(grad[x] + 2) * P]));
      // h_y over lines 3-5, h_x over 6-8, h_z over 9-11
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        o[(3 + d) * P] = mul2<T>(u[1], la[d]);
        o[(6 + d) * P] = mul2<T>(u[0], la[d]);
        o[(9 + d) * P] = mul2<T>(u[2], la[d]);
      }
    }
  }
  __syncthreads();
  // forward, both passes
  for (int it = threadIdx.x; it < npair * NF * R2; it += NT) {
    const int line = it / R2, j = it % R2;
    const C* b = s0 + line * P + j;
    C v[R1];
#pragma unroll
    for (int r = 0; r < R1; ++r) v[r] = b[r * R2];
    Dft<T, R1>::run(v);
    C* o = s1 + line * P + j * row;
#pragma unroll
    for (int r = 0; r < R1; ++r) o[r] = v[r];
  }
  __syncthreads();
  for (int it = threadIdx.x; it < npair * NF * R1; it += NT) {
    const int line = it / R1, j = it % R1;
    C u[R2];
    flex::load_column<T, R2, R1, row>(s1 + line * P + j, tw, j, u);
    Dft<T, R2>::run(u);
    C* o = s0 + line * P + j;
#pragma unroll
    for (int r = 0; r < R2; ++r) o[r * R1] = u[r];
  }
  __syncthreads();
  // half spectra of the two points of a pair, kept modes
  constexpr int NO = ADJ ? 9 : 3;
  for (int it = threadIdx.x; it < npair * NO * kz; it += NT) {
    int line, k;
    split_kz(a.g, it, &line, &k);
    const int pr = line / NO, l = line % NO;
    auto half = [&](int ln, C* e0, C* e1) {
      const C* b = s0 + (pr * NF + ln) * P;
      const C p = b[k], m = cconj(b[k == 0 ? 0 : N - k]);
      const T hs = T(0.5 * a.fwd) * (ADJ && k > 0 ? T(2) : T(1));
      const C df = csub(p, m);
      *e0 = cscale(cadd(p, m), hs);
      *e1 = mk<T>(df.y * hs, -df.x * hs);
    };
    C e0, e1;
    half(l, &e0, &e1);
    if (ADJ && l < 3) {
      C h0, h1;
      half(9 + l, &h0, &h1);
      const T k0 = T(-k * a.g.kscale);
      e0 = cadd(e0, ik<T>(k0, h0));
      e1 = cadd(e1, ik<T>(k0, h1));
    }
    const int64_t pt = 2 * static_cast<int64_t>(pair0 + pr);
    C* o = a.f + (static_cast<int64_t>(l) * a.points + pt) * kz + k;
    o[0] = e0;
    if (pt + 1 < a.points) o[kz] = e1;
  }
}

// The kernels of one axis length.
template <typename T>
struct Entry {
  int n, R1, R2;
  cudaError_t (*line[4])(const LineArgs<T>& a, int nf, cudaStream_t st);  // by LineKind
  cudaError_t (*z)(const ZArgs<T>& a, cudaStream_t st);
  cudaError_t (*z_adjoint)(const ZArgs<T>& a, cudaStream_t st);  // null: a pair does not fit shared memory
};
// The entries of one group of lengths (ns_lengths.h), defined by
// ns_lines_inst.cu in a translation unit each.
template <typename T, int GROUP>
struct Group {
  static const Entry<T>* entries(int* count);
};

}  // namespace nsl
}  // namespace dev
}  // namespace dfft
