"""Workloads of the distributed FFT package that its speed is judged by.

Every case is one pass of a user's program through the public entry points:
transforms there and back (``dfft.execute``), a transform with its gradient
(``dfft.autograd.fft``), many fields at once (``dfft.Batch``) and the
Navier-Stokes solver (``dfft.autograd.navier_stokes``).  Buffers hold the
local blocks of all ranks of a topology, concatenated in rank order.

Extents and topologies are written as texts, ``"512x512x512"`` and ``"4x4x1"``.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("distributed-fft-for-kokkos_b200"))

import dfft  # noqa: E402
import dfft.autograd  # noqa: E402

_REAL = {"float32": torch.float32, "float64": torch.float64}
_COMPLEX = {"float32": torch.complex64, "float64": torch.complex128}


def _ints(text):
    return tuple(int(p) for p in text.split("x"))


def _text(values):
    return "x".join(str(v) for v in values)


def _fft(name, extents, tin, tout, real=False, precision="float32", axes="0x1x2", layout="right", norm="backward",
         kind="roundtrip"):
    return {"name": name, "kind": kind, "extents": extents, "axes": axes, "in_topology": tin, "out_topology": tout,
            "real": real, "precision": precision, "layout": layout, "norm": norm}


def listed():
    return [
        # the smallest call: a field that fits a fraction of the chip, where
        # launches and the host path count (unit-test and debugging size)
        _fft("c2c_32_f64_slab", "32x32x32", "2x1x1", "1x2x1", precision="float64"),
        # the benchmark's own workload: a large complex64 field on a 4 x 4 pencil
        _fft("c2c_512_f32_pencil", "512x512x512", "4x4x1", "1x4x4"),
        # double precision, the package's default, at an everyday size
        _fft("c2c_256_f64_pencil", "256x256x256", "2x2x1", "1x2x2", precision="float64", norm="ortho"),
        # a large real field of a simulation code on slabs
        _fft("r2c_384_f64_slab", "384x384x384", "4x1x1", "1x4x1", real=True, precision="float64"),
        # a transform inside a training step: forward and gradient, ragged
        # half spectrum (129 modes over 2 ranks)
        _fft("grad_r2c_256_f32_pencil", "256x256x256", "2x2x1", "1x2x2", real=True, kind="grad"),
        # grids chosen by physics, not by powers of two: 2^a 3^b 5^c lengths,
        # ragged blocks
        _fft("c2c_smooth_f32_pencil", "300x250x360", "2x3x1", "1x2x3"),
        _fft("r2c_smooth_f64_slab", "200x180x252", "3x1x1", "1x3x1", real=True, precision="float64"),
        # arbitrary grids: prime lengths beside a smooth one
        _fft("r2c_any_f64_slab", "131x105x157", "2x1x1", "1x2x1", real=True, precision="float64"),
        # a stack of 2D transforms in Fortran order
        _fft("c2c_2d_left_f32", "256x192x128", "2x1x1", "1x2x1", axes="0x1", layout="left"),
        # one step of the solver on a turbulence grid: transforms and
        # pointwise kernels, 3 velocity components
        {"name": "ns_192_f32", "kind": "ns", "extents": "192x192x192", "topology": "2x2", "precision": "float32",
         "grad": False},
        # the same with the gradient of a loss, in double precision
        {"name": "ns_grad_96_f64", "kind": "ns", "extents": "96x96x96", "topology": "2x2", "precision": "float64",
         "grad": True},
        # many fields of uneven sizes at once (the benchmark's 16 fields)
        {"name": "batch_16_f32", "kind": "batch", "edges": "192x96x64x96x96x192x96x64x96x128x192x128x192x64x192x64",
         "in_topology": "2x2x1", "out_topology": "1x2x2", "precision": "float32"},
    ]


# lengths of 2^k and 3 * 2^k points, of small primes, and any
_POW = [16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512]
_SMOOTH = [n for n in range(20, 401) if math.gcd(n, 210 ** 9) == n]


def _edges(rng, pick, limit, least=4096):
    while True:
        e = [pick() for _ in range(3)]
        if least <= e[0] * e[1] * e[2] <= limit:
            return e


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pow", "pow", "pow", "smooth", "smooth", "any", "grad", "stack", "ns", "ns", "batch"])
    precision = rng.choice(["float32", "float64"])
    half = 1 if precision == "float32" else 2
    if kind == "batch":
        edges = [rng.choice([32, 48, 64, 96, 128, 192]) for _ in range(rng.randint(4, 16))]
        return {"kind": "batch", "edges": _text(edges), "in_topology": "2x2x1", "out_topology": "1x2x2",
                "precision": precision}
    if kind == "ns":
        grad = rng.random() < 0.4
        top = 96 if grad else 192
        e = _edges(rng, lambda: rng.choice([n for n in (32, 48, 60, 64, 80, 96, 100, 128, 144, 160, 192) if n <= top]),
                   top ** 3 // half if not grad else top ** 3)
        return {"kind": "ns", "extents": _text(e), "topology": rng.choice(["1x1", "2x2", "2x3", "4x1"]),
                "precision": precision, "grad": grad}
    real = rng.random() < 0.5
    slab = rng.random() < 0.4
    p, q = rng.randint(2, 4), rng.randint(2, 4)
    tin, tout = ((p, 1, 1), (1, p, 1)) if slab else ((p, q, 1), (1, p, q))
    axes, layout = "0x1x2", "right"
    if kind == "pow" or kind == "grad":
        # the volume is spread over the logarithm from a latency-bound call to
        # the largest field
        limit = _log_int(rng, 2 ** 15, (2 ** 27 if kind == "pow" else 2 ** 25) // half)
        e = _edges(rng, lambda: rng.choice(_POW), limit, limit // 8)
    elif kind == "smooth":
        limit = _log_int(rng, 2 ** 17, 27000000 // half)
        e = _edges(rng, lambda: rng.choice(_SMOOTH), limit, limit // 8)
    elif kind == "any":
        e = [_log_int(rng, 17, 160) for _ in range(3)]
    else:  # a stack of 2D transforms along the last axis
        e = [rng.choice(_POW[:9]), rng.choice(_POW[:9]), _log_int(rng, 8, 160)]
        axes, layout, real = "0x1", rng.choice(["left", "right"]), False
        tin, tout = (p, 1, 1), (1, p, 1)
    case = _fft("", _text(e), _text(tin), _text(tout), real, precision, axes, layout,
                rng.choice(["backward", "forward", "ortho"]), "grad" if kind == "grad" else "roundtrip")
    del case["name"]
    return case


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _field(extents, real, precision, gen):
    n = math.prod(extents)
    if real:
        return torch.rand(n, dtype=_REAL[precision], device="cuda", generator=gen) * 2 - 1
    return torch.randn(n, dtype=_COMPLEX[precision], device="cuda", generator=gen)


def _plan(extents, tin, tout, axes, real, precision, layout, norm):
    gout = list(extents)
    if real:
        gout[axes[-1]] = extents[axes[-1]] // 2 + 1
    return dfft.Plan(extents, gout, axes, tin, tout, real_input=real, precision=precision, layout=layout, norm=norm)


def _velocity(extents, precision, gen):
    """A smooth divergence-free velocity field of unit size, (3, nx, ny, nz)."""
    u = torch.randn((3,) + extents, dtype=torch.float64, device="cuda", generator=gen)
    k = _wavenumbers(extents, "cuda")
    ksq = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    uk = torch.fft.rfftn(u, dim=(1, 2, 3)) * torch.exp(-ksq / 32.0)
    safe = torch.where(ksq == 0, torch.ones_like(ksq), ksq)
    div = (k[0] * uk[0] + k[1] * uk[1] + k[2] * uk[2]) / safe
    uk = torch.stack([uk[a] - k[a] * div for a in range(3)])
    u = torch.fft.irfftn(uk, s=extents, dim=(1, 2, 3))
    return (u / u.abs().max()).to(_REAL[precision])


_NS = {"nu": 1.0 / 1600.0, "dt": 1e-3, "lx": 2.0}


def _ns_topologies(case):
    px, py = _ints(case["topology"])
    return (1, px, py, 1), (1, 1, px, py)


def prepare(case, seed):
    gen = _generator(seed)
    kind, precision = case["kind"], case["precision"]
    if kind == "ns":
        e = _ints(case["extents"])
        tin, tout = _ns_topologies(case)
        plan = dfft.Plan((3,) + e, (3,) + e[:2] + (e[2] // 2 + 1,), (1, 2, 3), tin, tout, real_input=True,
                         precision=precision)
        u0 = _to_blocks(_velocity(e, precision, gen), tin, "right")
        st = {"kind": kind, "ns": dfft.NavierStokes(plan, **_NS), "u0": u0, "grad": case["grad"]}
        if case["grad"]:
            u0.requires_grad_(True)
            st["g"] = _field((3,) + e, True, precision, gen)
        return st
    tin, tout = _ints(case["in_topology"]), _ints(case["out_topology"])
    if kind == "batch":
        edges = _ints(case["edges"])
        plans = [_plan((e,) * 3, tin, tout, (0, 1, 2), False, precision, "right", "backward") for e in edges]
        xs = [_field((e,) * 3, False, precision, gen) for e in edges]
        return {"kind": kind, "batch": dfft.Batch(plans), "xs": xs, "ys": [torch.empty_like(x) for x in xs],
                "zs": [torch.empty_like(x) for x in xs]}
    e = _ints(case["extents"])
    plan = _plan(e, tin, tout, _ints(case["axes"]), case["real"], precision, case["layout"], case["norm"])
    x = _field(e, case["real"], precision, gen)
    if kind == "grad":
        g = torch.randn(plan.buffer_elements("out"), dtype=_COMPLEX[precision], device="cuda", generator=gen)
        return {"kind": kind, "plan": plan, "x": x.requires_grad_(True), "g": g}
    y = torch.empty(plan.buffer_elements("out"), dtype=_COMPLEX[precision], device="cuda")
    return {"kind": kind, "plan": plan, "x": x, "y": y, "z": torch.empty_like(x)}


def run(state):
    kind = state["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "roundtrip":
        plan, x, y, z = state["plan"], state["x"], state["y"], state["z"]
        dfft.execute(plan, x, y, dfft.Direction.forward, stream=stream)
        dfft.execute(plan, y, z, dfft.Direction.backward, stream=stream)
        return [y, z]
    if kind == "grad":
        y = dfft.autograd.fft(state["x"], state["plan"])
        (gx,) = torch.autograd.grad(y, state["x"], state["g"])
        return [y.detach(), gx]
    if kind == "batch":
        batch, xs, ys, zs = state["batch"], state["xs"], state["ys"], state["zs"]
        batch.execute(xs, ys, dfft.Direction.forward, stream=stream)
        batch.execute(ys, zs, dfft.Direction.backward, stream=stream)
        return ys + zs
    u = dfft.autograd.navier_stokes(state["u0"], state["ns"], 1)
    if not state["grad"]:
        return [u]
    (gu,) = torch.autograd.grad(u, state["u0"], state["g"])
    return [u.detach(), gu]


def _volume_work(n_real, n_complex, real, precision):
    """Bytes of one transform (read once, written once) and its flops."""
    r = 4 if precision == "float32" else 8
    nbytes = (r * n_real if real else 2 * r * n_complex) + 2 * r * n_complex
    return nbytes, (2.5 if real else 5.0)


def work(case):
    kind, precision = case["kind"], case["precision"]
    r = 4 if precision == "float32" else 8
    if kind == "batch":
        sizes = [e ** 3 for e in _ints(case["edges"])]
        return {"bytes": sum(4 * 2 * r * n for n in sizes), "flops": sum(10.0 * n * math.log2(n) for n in sizes)}
    e = _ints(case["extents"])
    n = math.prod(e)
    if kind == "ns":
        # a right-hand side has 12 inverse and 3 forward scalar transforms, a
        # step four of them, and 3 transforms on either side; the gradient
        # passes as many back
        passes = 2 if case["grad"] else 1
        return {"bytes": passes * 2 * 3 * n * r, "flops": passes * (4 * 15 + 6) * 2.5 * n * math.log2(n)}
    axes = _ints(case["axes"])
    m = list(e)
    if case["real"]:
        m[axes[-1]] = e[axes[-1]] // 2 + 1
    nbytes, per = _volume_work(n, math.prod(m), case["real"], precision)
    return {"bytes": 2 * nbytes, "flops": 2 * per * n * math.log2(math.prod(e[a] for a in axes))}


# ---- 64-bit values, in plain torch -------------------------------------


def _bins(n, p):
    """(start, length) of the p blocks of an axis: the first n % p are longer."""
    out, start = [], 0
    for i in range(p):
        length = n // p + (1 if i < n % p else 0)
        out.append((start, length))
        start += length
    return out


def _rank_slices(shape, topology):
    bins = [_bins(n, p) for n, p in zip(shape, topology)]
    for r in range(math.prod(topology)):
        idx, rest = [], r
        for p in reversed(topology):
            idx.append(rest % p)
            rest //= p
        yield tuple(slice(b[i][0], b[i][0] + b[i][1]) for b, i in zip(bins, reversed(idx)))


def _to_blocks(a, topology, layout):
    parts = []
    for sl in _rank_slices(a.shape, topology):
        b = a[sl]
        parts.append((b if layout == "right" else b.permute(*reversed(range(b.dim())))).reshape(-1))
    return torch.cat(parts)


def _from_blocks(flat, shape, topology, layout):
    out = torch.empty(shape, dtype=flat.dtype, device=flat.device)
    start = 0
    for sl in _rank_slices(shape, topology):
        ext = [s.stop - s.start for s in sl]
        b = flat[start:start + math.prod(ext)]
        start += math.prod(ext)
        out[sl] = b.reshape(ext) if layout == "right" else b.reshape(ext[::-1]).permute(*reversed(range(len(ext))))
    return out


def _forward(x, axes, real, norm):
    return torch.fft.rfftn(x, dim=axes, norm=norm) if real else torch.fft.fftn(x, dim=axes, norm=norm)


def _backward(y, extents, axes, real, norm):
    if not real:
        return torch.fft.ifftn(y, dim=axes, norm=norm)
    if len(axes) > 1:
        y = torch.fft.ifftn(y, dim=axes[:-1], norm=norm)
    return torch.fft.irfft(y, n=extents[axes[-1]], dim=axes[-1], norm=norm)


def _exact_roundtrip(x, tin, tout, axes, real, layout, norm, extents):
    xg = _from_blocks(x.to(torch.float64 if real else torch.complex128), extents, tin, layout)
    y = _forward(xg, axes, real, norm)
    z = _backward(y, extents, axes, real, norm)
    return _to_blocks(y, tout, layout), _to_blocks(z, tin, layout)


def _wavenumbers(extents, device):
    ks = []
    for a, n in enumerate(extents):
        i = torch.arange(n // 2 + 1 if a == 2 else n, dtype=torch.float64, device=device)
        if a < 2:
            i = torch.where(2 * i < n, i, i - n)
        ks.append((i * (2.0 / _NS["lx"])).reshape([-1 if b == a else 1 for b in range(3)]))
    return ks


def _exact_ns(u0, extents):
    """One RK4 step of the pseudo-spectral solver (2/3-rule dealiasing, projection)."""
    k = _wavenumbers(extents, u0.device)
    cut = [(n // 2) * 2 // 3 for n in extents]
    scale = _NS["lx"] / 2.0
    keep = ((k[0].abs() * scale <= cut[0]) & (k[1].abs() * scale <= cut[1]) & (k[2] * scale <= cut[2])).to(torch.float64)
    ksq = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    inv = torch.where(ksq == 0, torch.zeros_like(ksq), 1.0 / torch.where(ksq == 0, torch.ones_like(ksq), ksq))

    def fwd(u):
        return _forward(u, (1, 2, 3), True, "backward")

    def bwd(uk):
        return _backward(uk, (3,) + extents, (1, 2, 3), True, "backward")

    def rhs(uk):
        u = bwd(uk)
        adv = sum(u[a] * bwd(1j * k[a] * uk) for a in range(3))
        r = -keep * fwd(adv) - _NS["nu"] * ksq * uk
        div = (k[0] * r[0] + k[1] * r[1] + k[2] * r[2]) * inv
        return torch.stack([r[a] - k[a] * div for a in range(3)])

    y0, h = keep * fwd(u0), _NS["dt"]
    k1 = h * rhs(y0)
    k2 = h * rhs(y0 + k1 / 2)
    k3 = h * rhs(y0 + k2 / 2)
    k4 = h * rhs(y0 + k3)
    return bwd(y0 + (k1 + 2 * k2 + 2 * k3 + k4) / 6)


def exact(case, seed):
    gen = _generator(seed)
    kind, precision = case["kind"], case["precision"]
    if kind == "ns":
        e = _ints(case["extents"])
        tin, _ = _ns_topologies(case)
        u0 = _velocity(e, precision, gen).to(torch.float64)
        if not case["grad"]:
            return [_to_blocks(_exact_ns(u0, e), tin, "right")]
        g = _from_blocks(_field((3,) + e, True, precision, gen).to(torch.float64), (3,) + e, tin, "right")
        u0.requires_grad_(True)
        u = _exact_ns(u0, e)
        (gu,) = torch.autograd.grad(u, u0, g)
        return [_to_blocks(u.detach(), tin, "right"), _to_blocks(gu, tin, "right")]
    tin, tout = _ints(case["in_topology"]), _ints(case["out_topology"])
    if kind == "batch":
        ys, zs = [], []
        for e in _ints(case["edges"]):
            x = _field((e,) * 3, False, precision, gen)
            y, z = _exact_roundtrip(x, tin, tout, (0, 1, 2), False, "right", "backward", (e,) * 3)
            ys.append(y)
            zs.append(z)
        return ys + zs
    e, axes, layout, norm, real = (_ints(case["extents"]), _ints(case["axes"]), case["layout"], case["norm"],
                                   case["real"])
    x = _field(e, real, precision, gen)
    if kind == "roundtrip":
        return list(_exact_roundtrip(x, tin, tout, axes, real, layout, norm, e))
    m = list(e)
    if real:
        m[axes[-1]] = e[axes[-1]] // 2 + 1
    g = torch.randn(math.prod(m), dtype=_COMPLEX[precision], device="cuda", generator=gen)
    xg = _from_blocks(x.to(torch.float64 if real else torch.complex128), e, tin, layout).requires_grad_(True)
    gg = _from_blocks(g.to(torch.complex128), m, tout, layout)
    y = _forward(xg, axes, real, norm)
    (gx,) = torch.autograd.grad(y, xg, gg)
    return [_to_blocks(y.detach(), tout, layout), _to_blocks(gx, tin, layout)]
