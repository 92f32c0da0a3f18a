"""Timed cases: what programs on this engine have it do, over the sizes, precisions and exponents of its configurations.

Two kinds of pass, both through the C ABI of include/maxlq.h, which a Fortran or C++ driver calls on its own host arrays:

  cg       mlq_state_load, mlq_state_iterate, mlq_state_store, mlq_state_R: a field in, `iters` iterations of the
           conjugate-gradient search from it, the field and its R out.  This is what a run of the search consists of.
  grad, R  mlq_grad_l2 and mlq_R_parts of a host field: the gradient check and the diagnostics.

A context is what such a program keeps over all its fields, so one context serves every state of a case.  Fields are seeded Gaussian Fourier modes |j|^-slope exp(-(|j|/k0)^2),
divergence-free and 2/3-dealiased, the configurations' initial data.  In mixed precision the state on the device is FP32, so
the program keeps it as FP32 too; FP64 runs keep all bits.  At q != 4 in mixed precision the search follows FP32 noise of
the trial values, so its trajectory is not reproducible to more than about 1e-4; those runs are listed in FP64.
"""
import ctypes
import math

import numpy as np
import torch

import maxlq_b200 as mlq

# sizes are even, 2^a 3^b: the ones that the configurations name, their neighbours, and ragged ones with several factors 3
_SIZES = (32, 48, 64, 96, 128, 192, 256, 384, 512)
_RAGGED = (54, 72, 108, 144, 162, 216)


def listed():
    def cg(n, q, B, precision, iters, k0, slope=2.0):
        return {"name": f"cg_{n}_q{q:g}_{precision}_{iters}", "kind": "cg", "n": n, "q": q, "B": B, "precision": precision,
                "iters": iters, "k0": k0, "slope": slope}

    return [
        cg(32, 4.0, 1.0, "fp64", 10, 2.0),     # the smallest runs: a coarse start of a continuation
        cg(48, 8.0, 2.0, "fp64", 3, 3.0),      # a small instance of the many-instance sweep over N, q and B
        cg(64, 4.0, 1.0, "fp64", 10, 4.0),     # the plain 64^3 configuration
        cg(96, 6.0, 2.0, "fp64", 3, 6.0),      # sweep instance, N not a power of two
        cg(128, 3.0, 1.0, "fp64", 3, 8.0),     # sweep instance on the unit-vector branch (q < 4)
        cg(192, 4.0, 1.0, "mixed", 5, 8.0),    # a refinement between the powers of two
        cg(256, 4.0, 1.0, "fp64", 5, 8.0),     # the FP64 continuation size
        cg(256, 6.0, 4.0, "fp64", 2, 8.0),     # a higher exponent at that size
        cg(512, 4.0, 1.0, "mixed", 10, 16.0),  # the headline workload
        # one step at a time between the host and the device, for a driver that owns the loop
        cg(256, 4.0, 1.0, "mixed", 1, 8.0),
        # the L2 gradient for a gradient check
        {"name": "grad_128_q6_fp64", "kind": "grad", "n": 128, "q": 6.0, "B": 2.0, "precision": "fp64", "k0": 8.0,
         "slope": 5.0 / 3.0},
        # R of a host field at the Taylor-test configuration
        {"name": "R_512_q6_mixed", "kind": "R", "n": 512, "q": 6.0, "B": 4.0, "precision": "mixed", "k0": 16.0,
         "slope": 5.0 / 3.0},
    ]


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        n = rng.choice(_SIZES if rng.random() < 0.8 else _RAGGED)
        kind = rng.choice(("cg", "cg", "cg", "cg", "cg", "grad", "R"))
        case = {"kind": kind, "n": n, "q": rng.choice((3.0, 4.0, 4.0, 6.0, 8.0)),
                "B": round(math.exp(rng.uniform(math.log(0.5), math.log(8.0))), 3),
                "precision": rng.choice(("fp64", "mixed")), "k0": round(n / rng.uniform(12.0, 32.0), 3),
                "slope": rng.choice((5.0 / 3.0, 2.0))}
        if kind == "cg" and case["q"] != 4.0:
            case["precision"] = "fp64"
        if kind == "grad":
            case["precision"] = "fp64"  # what a gradient check needs
        if kind == "cg":
            case["iters"] = rng.randint(1, 5)
        if _cost(case) <= most and (n < 512 or case["precision"] == "mixed"):
            return case


def _real(case):
    return torch.float64 if case["precision"] == "fp64" else torch.float32


def _cut(n):
    """Largest |j| with 2 pi j <= 2 pi n / 3, as the dealiasing compares them."""
    pi = 4.0 * math.atan2(1.0, 1.0)
    return max(j for j in range(n // 2 + 1) if not 2.0 * pi * j > 2.0 * pi * float(n) / 3.0)


def _wave(n):
    """Integer wavenumbers (z, y, x) of the half spectrum, broadcastable."""
    f = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")
    x = torch.arange(n // 2 + 1, dtype=torch.float64, device="cuda")
    return f[:, None, None], f[None, :, None], x[None, None, :]


def _band(n, cut):
    z, y, x = _wave(n)
    return (z.abs() <= cut) & (y.abs() <= cut) & (x <= cut)


def _field(case, seed):
    """The seeded field on the GPU, (3, n, n, n) FP64, L2 norm B."""
    n = case["n"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    z, y, x = _wave(n)
    k2 = (z * z + y * y + x * x).clamp_(min=1.0)
    amp = k2 ** (-0.5 * case["slope"]) * torch.exp(-k2 / case["k0"] ** 2) * _band(n, _cut(n))
    amp[0, 0, 0] = 0.0
    h = [torch.fft.rfftn(torch.randn((n, n, n), dtype=torch.float64, device="cuda", generator=gen)).mul_(amp)
         for _ in range(3)]
    del amp
    div = (x * h[0] + y * h[1] + z * h[2]) / k2
    u = torch.empty((3, n, n, n), dtype=torch.float64, device="cuda")
    for c, k in enumerate((x, y, z)):
        u[c] = torch.fft.irfftn(h[c] - k * div, s=(n, n, n))
    u *= case["B"] / u.square().sum().div(float(n) ** 3).sqrt()
    return u


class _Context:
    def __init__(self, case):
        self.lib = mlq.load_library()
        p = mlq.default_params(case["n"], case["q"], case["B"], precision=case["precision"], optim_tol=0.0)
        self.ptr = ctypes.c_void_p()
        self.check(self.lib.mlq_init(ctypes.byref(self.ptr), ctypes.byref(p)))

    def check(self, status):
        if status != mlq.MLQ_OK:
            raise mlq.MlqError(status, str(self.lib.mlq_last_error(self.ptr)))

    def __del__(self):
        if self.ptr:
            self.lib.mlq_finalize(self.ptr)


# the ways in which a search ends, all of them results
_ENDS = (mlq.MLQ_OK, mlq.MLQ_ERR_MNBRAK_UPHILL, mlq.MLQ_ERR_MNBRAK_ITMAX, mlq.MLQ_ERR_TAU_MAX, mlq.MLQ_ERR_J_DECREASED)
_kept = {}


def _context(case):
    key = (case["n"], case["q"], case["B"], case["precision"])
    if key not in _kept:
        _kept.clear()
        _kept[key] = _Context(case)
    return _kept[key]


def prepare(case, seed):
    u = _field(case, seed)
    host = torch.empty(u.shape, dtype=torch.float64, pin_memory=True)
    host.copy_(u)
    del u
    torch.cuda.empty_cache()
    state = {"case": case, "u": host.numpy(), "host": host}
    if case["kind"] != "R":
        state["out"] = torch.empty(host.shape, dtype=torch.float64, pin_memory=True)
    if case["kind"] == "cg" and case["precision"] == "mixed":
        state["kept"] = torch.empty(host.shape, dtype=torch.float32)
    state["ctx"] = _context(case)
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    lib, h, u = ctx.lib, ctx.ptr, mlq.dptr(state["u"])
    J = []

    @mlq.ITER_CB
    def record(info, _):
        J.append(info.contents.J1)

    done = ctypes.c_int(0)
    if case["kind"] == "cg":
        ctx.check(lib.mlq_state_load(h, u))
        status = lib.mlq_state_iterate(h, case["iters"], record, None, ctypes.byref(done))
        if status not in _ENDS:
            ctx.check(status)
        ctx.check(lib.mlq_state_store(h, mlq.dptr(state["out"].numpy())))
        parts = np.zeros(3)
        norm = ctypes.c_double(0.0)
        ctx.check(lib.mlq_state_R(h, mlq.dptr(parts), ctypes.byref(norm)))
        u_out = state["kept"].copy_(state["out"]) if "kept" in state else state["out"]
        return {"u": u_out, "J": torch.tensor(J, dtype=_real(case)),
                "R": torch.tensor(parts, dtype=_real(case)), "norm": norm.value}
    if case["kind"] == "grad":
        ctx.check(lib.mlq_grad_l2(h, u, mlq.dptr(state["out"].numpy())))
        return {"grad": state["out"]}
    parts = np.zeros(3)
    ctx.check(lib.mlq_R_parts(h, u, mlq.dptr(parts)))
    return {"R": torch.tensor(parts, dtype=_real(case))}


def _iterations(case):
    return case["iters"] if case["kind"] == "cg" else 0


def _transforms(case):
    """Real 3D transforms of a pass: in and out, and 51 per iteration at q = 4 (15 forward, 36 inverse); elsewhere each
    of some 13 trials adds the transform of one power of |u|.  A gradient is 20, R alone 18."""
    if case["kind"] == "cg":
        return 6 + _iterations(case) * (51 if case["q"] == 4.0 else 64)
    return 3 + (20 if case["kind"] == "grad" else 18)


def work(case):
    n3 = float(case["n"]) ** 3
    width = 8 if case["precision"] == "fp64" else 4
    out = {"cg": 3 * width, "grad": 3 * width, "R": 0}[case["kind"]]
    modes = (2 * _cut(case["n"]) + 1) ** 2 * (_cut(case["n"]) + 1)
    # an iteration reads and writes the state, its gradient and the two transported vectors
    state = 8 * 3 * modes * 2 * width * _iterations(case) if case["kind"] == "cg" else 0
    return {"bytes": n3 * (24 + out) + state, "flops": _transforms(case) * 2.5 * n3 * math.log2(n3)}


def _cost(case):
    """Rough time of a pass, for draw(): its transforms, and at q != 4 all of those of the trials."""
    many = 12.0 if case["kind"] == "cg" and case["q"] != 4.0 else 1.0
    slow = 4.0 if case["n"] % 3 == 0 else 1.0
    return work(case)["flops"] * many * slow * (2.0 if case["precision"] == "fp64" else 1.0)


# ---- the values in 64 bits -----------------------------------------------------------------------------------------

_TINY = 2.0e-16


class _Plain:
    """R and its L2 gradient as their formulas read, with torch's FFTs."""

    def __init__(self, n, q):
        self.n, self.q = n, q
        two_pi = 2.0 * math.pi
        self.k = [two_pi * f for f in reversed(_wave(n))]  # x, y, z
        self.k2 = self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2

    def hat(self, f):
        return torch.fft.rfftn(f)

    def phys(self, h):
        return torch.fft.irfftn(h, s=(self.n,) * 3)

    def cut(self, f, order=2.0):
        c = max(j for j in range(self.n // 2 + 1) if not 2.0 * math.pi * j > 2.0 * math.pi * float(self.n) / (order + 1.0))
        return f if c >= self.n // 2 else self.phys(self.hat(f) * _band(self.n, c))

    def grad(self, f):
        h = self.hat(f)
        return [self.phys(1j * k * h) for k in self.k]

    def inv_lap(self, f):
        h = -self.hat(f) / self.k2.clamp(min=1.0)
        h[0, 0, 0] = 0.0
        return self.phys(h)

    def lap(self, f):
        return self.phys(-self.k2 * self.hat(f))

    def power(self, g, k):
        if k + _TINY < 0.0:
            return torch.where(g.abs() < _TINY, torch.zeros_like(g), g ** k)
        if k + _TINY < 2.0:
            return self.cut(g ** k, k)
        return self.cut(self.cut(g * g) * self.power(g, k - 2.0))

    def setup(self, u):
        self.u = u
        self.g = sum(c * c for c in u)
        s = self.cut(self.g)
        self.g = s.clamp(min=0.0).sqrt()
        self.unit = self.q < 4.0 - _TINY
        n = s.abs().sqrt()
        self.v = [torch.where(n < _TINY, torch.zeros_like(c), c / n) for c in u] if self.unit else list(u)
        self.du = [self.grad(c) for c in u]  # du[i][j] = d_j u_i
        self.a2 = self.power(self.g, self.q - 2.0)
        self.mult = self.a2 if self.unit else self.power(self.g, self.q - 4.0)
        self.p = self.inv_lap(-self.cut(sum(self.du[i][j] * self.du[j][i] for i in range(3) for j in range(3))))

    def R(self, u):
        self.setup(u)
        q = self.q

        def mean(a, b):
            return float((a * b).mean())

        r1 = -mean(self.a2, self.cut(sum(d * d for row in self.du for d in row)))
        w = [self.cut(sum(self.v[i] * self.du[i][j] for i in range(3))) for j in range(3)]
        r2 = -(q - 2.0) * mean(self.mult, self.cut(sum(x * x for x in w)))
        r3 = (q - 2.0) * mean(self.cut(self.p * self.mult), self.cut(sum(a * b for a, b in zip(self.v, w))))
        h = self.power(self.g, q / 2.0)
        return [r1 + r2 + r3, r1 + r2, r3], mean(h, h) ** (1.0 / q)

    def gradient(self, u):
        self.setup(u)
        q, cut = self.q, self.cut
        gp, lap = self.grad(self.p), [self.lap(c) for c in u]
        t = cut(sum(self.v[i] * (lap[i] - gp[i]) for i in range(3)))
        t = cut(self.mult * t)
        c = [cut(self.a2 * x) for x in u]
        h = sum(1j * k * self.hat(x) for k, x in zip(self.k, c))
        ga = self.grad(self.inv_lap(self.phys(h)))
        out = []
        for i in range(3):
            z = (q - 2.0) * t * self.v[i] - self.a2 * gp[i] + 2.0 * sum(self.du[k][i] * ga[k] for k in range(3))
            out.append(cut(z + self.a2 * lap[i]) + self.lap(c[i]))
        return torch.stack(out)


def exact(case, seed):
    u = _field(case, seed)
    plain = _Plain(case["n"], case["q"])
    if case["kind"] == "grad":
        return {"grad": plain.gradient(u)}
    if case["kind"] == "R":
        return {"R": torch.tensor(plain.R(u)[0], dtype=torch.float64)}
    return None  # where a line search ends depends on its tolerance, not on the formulas alone
