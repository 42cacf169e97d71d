// Host side of the Navier-Stokes line kernels: geometry, work buffers, the
// launch sequence of a right-hand side and of its adjoint, and the pointwise
// steps that end them.
#include "ns_lines.hpp"

#include <algorithm>
#include <map>
#include <string>
#include <vector>

#include "ns_lines.cuh"
#include "plan.hpp"

namespace dfft {
namespace dev {
namespace nsl {
namespace {

// wavenumbers of kept point t of (kx, ky, kz)
struct Wave {
  double kx, ky, kz, ksq, inv;
};
__device__ __forceinline__ Wave wave_of(const Grid& g, int t) {
  int xy, iz;
  split_kz(g, t, &xy, &iz);
  const int ix = xy / g.y.k, iy = xy - ix * g.y.k;
  Wave w;
  w.kx = mode(g.x, ix) * g.kscale;
  w.ky = mode(g.y, iy) * g.kscale;
  w.kz = iz * g.kscale;
  w.ksq = w.kx * w.kx + w.ky * w.ky + w.kz * w.kz;
  w.inv = t == 0 ? 0.0 : 1.0 / w.ksq;
  return w;
}

template <typename T>
struct UpdateArgs {
  Grid g;
  int total;  // kx ky kz
  const cplx<T>* adv;
  const cplx<T>* u;  // state the right-hand side is taken at
  cplx<T>* out;
  const cplx<T>* y0;
  cplx<T> *k1, *k2, *k3;
  double nu, h;
};

// f = P(-adv - nu k^2 u) and what STEP does with it: 0 .. 3 the stages of the
// low-storage RK4 (y0, k1, k2, k3 kept; the next state to out), 4 out = f, 5
// out = y0 + h f.  In place (out = u) too: a point is read and written by one
// thread.
template <typename T, int STEP>
__global__ void __launch_bounds__(256) ns_update_kernel(const __grid_constant__ UpdateArgs<T> a) {
  using C = cplx<T>;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.total) return;
  const Wave w = wave_of(a.g, t);
  const T visc = T(-a.nu * w.ksq), ikk = T(w.inv), hh = T(a.h);
  const T kk[3] = {T(w.kx), T(w.ky), T(w.kz)};
  C r[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const C v = a.adv[static_cast<int64_t>(d) * a.total + t], um = a.u[static_cast<int64_t>(d) * a.total + t];
    r[d] = mk<T>(-v.x + visc * um.x, -v.y + visc * um.y);
  }
  const C div = mk<T>((kk[0] * r[0].x + kk[1] * r[1].x + kk[2] * r[2].x) * ikk,
                      (kk[0] * r[0].y + kk[1] * r[1].y + kk[2] * r[2].y) * ikk);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int64_t e = static_cast<int64_t>(d) * a.total + t;
    const C f = mk<T>(r[d].x - kk[d] * div.x, r[d].y - kk[d] * div.y);
    const C hf = mk<T>(f.x * hh, f.y * hh);
    if (STEP == 4) {
      a.out[e] = f;
      continue;
    }
    const C y = a.y0[e];
    if (STEP == 0) a.k1[e] = hf;
    if (STEP == 1) a.k2[e] = hf;
    if (STEP == 2) a.k3[e] = hf;
    if (STEP == 0 || STEP == 1) {
      a.out[e] = mk<T>(y.x + hf.x / T(2), y.y + hf.y / T(2));
    } else if (STEP == 3) {
      const C p = a.k1[e], q = a.k2[e], s = a.k3[e];
      a.out[e] = mk<T>(y.x + (p.x + T(2) * q.x + T(2) * s.x + hf.x) / T(6),
                       y.y + (p.y + T(2) * q.y + T(2) * s.y + hf.y) / T(6));
    } else {
      a.out[e] = mk<T>(y.x + hf.x, y.y + hf.y);
    }
  }
}

// adjoint: g = -nu k^2 mu + S - i k_x Hx, fields S and Hx in `in`, and the
// backward stage of the RK4 step (NsLines::Vjp): with the projection of the
// next cotangent, one pass where g, two or three sums and the projection were
// five (step and gradient at 96^3 FP64: 15 launches fewer, 1270 -> 1216 us).
template <typename T>
struct AdjointArgs {
  Grid g;
  int total;
  const cplx<T>* in;
  cplx<T>* mu;
  cplx<T>* out;
  const cplx<T>* l;
  cplx<T>* ly0;
  double nu, h, direct, up;
  int first;
};

template <typename T>
__device__ __forceinline__ void project_point(const Wave& w, cplx<T>* v) {
  const T ikk = T(w.inv);
  const T kk[3] = {T(w.kx), T(w.ky), T(w.kz)};
  const cplx<T> div = mk<T>((kk[0] * v[0].x + kk[1] * v[1].x + kk[2] * v[2].x) * ikk,
                            (kk[0] * v[0].y + kk[1] * v[1].y + kk[2] * v[2].y) * ikk);
#pragma unroll
  for (int d = 0; d < 3; ++d) v[d] = mk<T>(v[d].x - kk[d] * div.x, v[d].y - kk[d] * div.y);
}

template <typename T>
__global__ void __launch_bounds__(256) ns_adjoint_update_kernel(const __grid_constant__ AdjointArgs<T> a) {
  using C = cplx<T>;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.total) return;
  const Wave w = wave_of(a.g, t);
  const T visc = T(-a.nu * w.ksq), kx = T(-w.kx), hh = T(a.h);
  C c[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int64_t e = static_cast<int64_t>(d) * a.total + t;
    const C m = a.mu[e], s = cadd(a.in[e], ik<T>(kx, a.in[e + static_cast<int64_t>(3) * a.total]));
    const C g = mk<T>(visc * m.x + s.x, visc * m.y + s.y);
    if (a.out) {
      a.out[e] = g;
      continue;
    }
    const C l = a.l[e], y = a.first ? l : a.ly0[e];
    a.ly0[e] = mk<T>(y.x + hh * g.x, y.y + hh * g.y);
    const T di = T(a.direct), hu = T(a.h * a.up);
    c[d] = mk<T>(di * l.x + hu * g.x, di * l.y + hu * g.y);
  }
  if (a.out || a.direct == 0.0) return;
  project_point<T>(w, c);
#pragma unroll
  for (int d = 0; d < 3; ++d) a.mu[static_cast<int64_t>(d) * a.total + t] = c[d];
}

// mu = P(s c)
template <typename T>
__global__ void __launch_bounds__(256)
    ns_kept_project_kernel(const Grid g, int total, const cplx<T>* c, cplx<T>* mu, double s) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  cplx<T> v[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) v[d] = cscale(c[static_cast<int64_t>(d) * total + t], T(s));
  project_point<T>(wave_of(g, t), v);
#pragma unroll
  for (int d = 0; d < 3; ++d) mu[static_cast<int64_t>(d) * total + t] = v[d];
}

template <typename T, int... G>
std::map<int, Entry<T>> all_entries() {
  std::map<int, Entry<T>> all;
  auto add = [&](const Entry<T>* (*get)(int*)) {
    int n = 0;
    const Entry<T>* e = get(&n);
    for (int i = 0; i < n; ++i) all.emplace(e[i].n, e[i]);
  };
  (add(&Group<T, G>::entries), ...);
  return all;
}

template <typename T>
const Entry<T>* find_entry(int n) {
  static const std::map<int, Entry<T>> table = all_entries<T, 0, 1, 2, 3>();
  const auto it = table.find(n);
  return it == table.end() ? nullptr : &it->second;
}

}  // namespace
}  // namespace nsl
}  // namespace dev

namespace {

using namespace dev;
using namespace dev::nsl;

void ck(cudaError_t e, const char* what) {
  if (e != cudaSuccess) fail(kErrCuda, std::string(what) + ": " + cudaGetErrorString(e));
}

template <typename T>
class Lines final : public NsLines {
  using C = cplx<T>;

 public:
  bool init(int nx, int ny, int nz, int cx, int cy, int cz, double kscale, double bs, double fs) {
    back_ = bs;
    fwd_ = fs;
    g_.kscale = kscale;
    if (!axis(g_.x, &ex_, nx, cx, 2 * cx + 1) || !axis(g_.y, &ey_, ny, cy, 2 * cy + 1) ||
        !axis(g_.z, &ez_, nz, cz, cz + 1) || !ez_->z)
      return false;
    const long long kz = g_.z.k, most = (1ll << 31) - 1;
    // the kernels index lines, and elements along one, with 32 bits
    if (static_cast<long long>(nx) * ny > most || nx * kz > most || static_cast<long long>(nx) * g_.y.k * kz > most ||
        static_cast<long long>(g_.x.k) * ny * kz > most)
      return false;
    g_.magic_kz = kz > 1 ? static_cast<unsigned>(((1ull << 32) + kz - 1) / kz) : 0;
    return true;
  }

  void alloc() {
    x_ = dmalloc(9 * xq());
    y_ = dmalloc(9 * xyz());
    for (auto ax : {std::make_pair(&g_.x, ex_), std::make_pair(&g_.y, ey_), std::make_pair(&g_.z, ez_)}) {
      const std::vector<double> h = two_pass_twiddles(ax.second->R1, ax.second->R2, false);
      const std::vector<T> t(h.begin(), h.end());
      C* p = dmalloc(static_cast<std::size_t>(ax.first->n));
      ck(cudaMemcpy(p, t.data(), t.size() * sizeof(T), cudaMemcpyHostToDevice), "ns twiddles");
      ax.first->tw = p;
    }
  }

  ~Lines() override {
    for (void* p : owned_) cudaFree(p);
  }

  std::size_t elements() const override { return 3 * static_cast<std::size_t>(kept_points()); }
  bool adjoint_supported() const override { return ez_->z_adjoint != nullptr; }
  void adjoint_alloc() override {
    if (!lambda_) lambda_ = dmalloc(3 * xyz());
  }

  void rhs(const Update& w, cudaStream_t st) override {
    back_fields(static_cast<const C*>(w.u), st);
    z_stage(false, st);
    line(kYForward, y_, x_, 1, 0, st);
    line(kXForward, x_, y_, 1, 0, st);
    UpdateArgs<T> a{g_, kept_points(), y_, static_cast<const C*>(w.u), static_cast<C*>(w.out),
                    static_cast<const C*>(w.y0), static_cast<C*>(w.k1), static_cast<C*>(w.k2), static_cast<C*>(w.k3),
                    w.nu, w.h};
    const unsigned grid = static_cast<unsigned>((kept_points() + 255) / 256);
    switch (w.step) {
      case 0: ns_update_kernel<T, 0><<<grid, 256, 0, st>>>(a); break;
      case 1: ns_update_kernel<T, 1><<<grid, 256, 0, st>>>(a); break;
      case 2: ns_update_kernel<T, 2><<<grid, 256, 0, st>>>(a); break;
      case 3: ns_update_kernel<T, 3><<<grid, 256, 0, st>>>(a); break;
      case 4: ns_update_kernel<T, 4><<<grid, 256, 0, st>>>(a); break;
      default: ns_update_kernel<T, 5><<<grid, 256, 0, st>>>(a); break;
    }
    ck(cudaGetLastError(), "ns update");
  }

  void vjp(const Vjp& w, cudaStream_t st) override {
    adjoint_alloc();
    back_fields(static_cast<const C*>(w.y), st);
    line(kXInverse, static_cast<const C*>(w.mu), x_, 1, 0, st);
    line(kYInverse, x_, lambda_, 1, 0, st);
    z_stage(true, st);
    line(kYForward, y_, x_, 3, 0, st);
    line(kXForward, x_, y_, 2, 1, st);
    const AdjointArgs<T> a{g_, kept_points(), y_, static_cast<C*>(w.mu), static_cast<C*>(w.out),
                           static_cast<const C*>(w.l), static_cast<C*>(w.ly0), w.nu, w.h, w.direct, w.up,
                           w.first ? 1 : 0};
    ns_adjoint_update_kernel<T><<<static_cast<unsigned>((kept_points() + 255) / 256), 256, 0, st>>>(a);
    ck(cudaGetLastError(), "ns adjoint update");
  }

  void project(const void* c, void* mu, double s, cudaStream_t st) override {
    ns_kept_project_kernel<T><<<static_cast<unsigned>((kept_points() + 255) / 256), 256, 0, st>>>(
        g_, kept_points(), static_cast<const C*>(c), static_cast<C*>(mu), s);
    ck(cudaGetLastError(), "ns projection");
  }

 private:
  Grid g_{};
  const Entry<T>*ex_ = nullptr, *ey_ = nullptr, *ez_ = nullptr;
  double back_ = 1.0, fwd_ = 1.0;
  // x_: fields over (nx, ky, kz), y_: over (nx, ny, kz); up to 9 of each
  C *x_ = nullptr, *y_ = nullptr, *lambda_ = nullptr;
  std::vector<void*> owned_;

  int kept_points() const { return g_.x.k * g_.y.k * g_.z.k; }
  std::size_t xq() const { return static_cast<std::size_t>(g_.x.n) * g_.y.k * g_.z.k; }
  std::size_t xyz() const { return static_cast<std::size_t>(g_.x.n) * g_.y.n * g_.z.k; }

  C* dmalloc(std::size_t n) {
    void* p = nullptr;
    ck(cudaMalloc(&p, n * sizeof(C)), "ns alloc");
    owned_.push_back(p);
    return static_cast<C*>(p);
  }

  static bool axis(Axis& a, const Entry<T>** e, int n, int c, int k) {
    a.n = n;
    a.c = c;
    a.k = k;
    *e = find_entry<T>(n);
    return *e != nullptr && k <= n;
  }

  void line(LineKind kind, const C* in, C* out, int nf, int adjoint, cudaStream_t st) {
    const bool x = kind == kXInverse || kind == kXForward;
    LineArgs<T> a{g_, in, out, x ? g_.y.k * g_.z.k : g_.x.n * g_.z.k, adjoint};
    ck((x ? ex_ : ey_)->line[kind](a, nf, st), "ns lines");
  }

  // U and V along x, then U, i k_y U and V along y
  void back_fields(const C* u, cudaStream_t st) {
    line(kXInverse, u, x_, 2, 0, st);
    line(kYInverse, x_, y_, 3, 0, st);
  }

  // (adjoint: B^H is 2 R2C backward_scale on the interior modes, lambda = F^H(-mu))
  void z_stage(bool adjoint, cudaStream_t st) {
    const ZArgs<T> a{g_, y_, lambda_, g_.x.n * g_.y.n, back_, adjoint ? back_ : fwd_, -fwd_};
    ck(adjoint ? ez_->z_adjoint(a, st) : ez_->z(a, st), "ns z lines");
  }
};

template <typename T>
std::unique_ptr<NsLines> make(int nx, int ny, int nz, int cx, int cy, int cz, double kscale, double bs, double fs) {
  auto p = std::make_unique<Lines<T>>();
  if (!p->init(nx, ny, nz, cx, cy, cz, kscale, bs, fs)) return nullptr;
  p->alloc();
  return p;
}

}  // namespace

std::unique_ptr<NsLines> NsLines::create(bool dbl, int nx, int ny, int nz, int cx, int cy, int cz, double kscale,
                                         double backward_scale, double forward_scale) {
  return dbl ? make<double>(nx, ny, nz, cx, cy, cz, kscale, backward_scale, forward_scale)
             : make<float>(nx, ny, nz, cx, cy, cz, kscale, backward_scale, forward_scale);
}

}  // namespace dfft
