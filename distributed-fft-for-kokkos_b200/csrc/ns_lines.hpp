// Host side of the Navier-Stokes line kernels (ns_lines.cuh): the right-hand
// side and its adjoint on spectra of kept modes, (3, kx, ky, kz) in C order.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <memory>

namespace dfft {

class Plan;

class NsLines {
 public:
  // null if the kernels do not take the grid: every axis length must have
  // kernels (ns_lengths.h) and a pair of z lines fit one CTA's shared memory
  // (backward_scale / forward_scale: the plan's normalisation)
  static std::unique_ptr<NsLines> create(bool dbl, int nx, int ny, int nz, int cx, int cy, int cz, double kscale,
                                         double backward_scale, double forward_scale);
  virtual ~NsLines() = default;

  // elements of one spectrum of kept modes
  virtual std::size_t elements() const = 0;
  // the adjoint's z kernel fits as well
  virtual bool adjoint_supported() const = 0;
  // buffers the adjoint needs (allocated on the first call)
  virtual void adjoint_alloc() = 0;
  // f(u) = P(-adv - nu k^2 u) and what `step` does with it: 0 .. 3 the stages of
  // the low-storage RK4, 4 out = f, 5 out = y0 + h f
  struct Update {
    const void* u = nullptr;
    void* out = nullptr;
    const void* y0 = nullptr;
    void *k1 = nullptr, *k2 = nullptr, *k3 = nullptr;
    double nu = 0.0, h = 0.0;
    int step = 4;
  };
  virtual void rhs(const Update& w, cudaStream_t st) = 0;
  // g = (d f / d u at y)^T c with mu = P c given, and what becomes of it
  struct Vjp {
    const void* y = nullptr;
    void* mu = nullptr;
    double nu = 0.0;
    void* out = nullptr;  // out = g; or, null, one stage of an RK4 step backwards:
    // ly0 <- (first: l, else ly0) + h g, and, if direct != 0, the next stage's
    // mu <- P(direct l + h up g)
    const void* l = nullptr;
    void* ly0 = nullptr;
    double h = 0.0, direct = 0.0, up = 0.0;
    bool first = false;
  };
  virtual void vjp(const Vjp& w, cudaStream_t st) = 0;
  // mu = P(s c)
  virtual void project(const void* c, void* mu, double s, cudaStream_t st) = 0;
};

}  // namespace dfft
