"""The work a program asks of deft_gb300, as cases that can be timed and checked.

A case is a dict of plain values.  `listed` names the standing ones, `draw`
gives more of the same ranges, `prepare` makes what a program holds before the
call (fields on the GPU, grids, functionals, minimisers, a network), `run` is
one pass through the public entry points (the C ABI of include/deft_gb300.h
through deft_gb300._lib, and deft_gb300.warmstart), `work` what the pass cannot
do without, and `exact` its outputs by plain torch in 64 bits.

Families (`case["do"]`):
  energy_grad  one Functional::integral + integralgrad on device fields
  solve        a minimisation from a given start to |grad F| < gtol
  warm_solve   network forward pass, checked start, mixed-precision solve
  batch        many independent solves from host arrays in one call
  network      forward pass of the warm-start network, with "grad" also the
               loss and its parameter gradient (one training sample)
"""
import ctypes
import math
import os

import numpy as np
import torch

from deft_gb300 import _lib
from deft_gb300.api import default_context
from deft_gb300.warmstart import FourierOperator, solve_batch

DEV = "cuda:0"
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(_lib.__file__)), "weights",
                       "fno_wb128_2000.bf16")

# liquid water in atomic units: radius, kT, density and the association and
# dispersion parameters (epsilon_a, kappa_a, epsilon_d, lambda_d, length scaling)
KB, ANGSTROM = 3.16681539628059e-6, 1.8897261
WATER_R, WATER_KT, WATER_N = 3.03420 * ANGSTROM / 2, 298.15 * KB, 4.9388942e-3
WATER_MU = 0.0176131572
WATER = (1400.0 * KB, 0.0381876 * (3.03420 * ANGSTROM) ** 3, 250.0 * KB, 1.78890, 0.353)


# ---------------------------------------------------------------------------
# The cases

def listed():
    return [
        # a small slit, the size of the quick-start and of most unit problems:
        # launches and the wait for the result are all there is
        {"name": "slit_32", "do": "energy_grad", "hs": "wb", "nx": 32, "ny": 32, "nz": 32,
         "dx": 0.2, "eta": 0.3, "mixed": False, "veff": False, "vext": False, "fcc": False},
        # the memory test's cell: face-centred cubic, 77^3, effective potential
        # as the variable, gradient and preconditioned gradient
        {"name": "fcc_veff_77", "do": "energy_grad", "hs": "wb", "nx": 77, "ny": 77, "nz": 77,
         "dx": 0.2, "eta": 0.3, "mixed": False, "veff": True, "vext": False, "fcc": True},
        # the usual production grid, mark II with an external potential
        {"name": "mark2_vext_128", "do": "energy_grad", "hs": "m2", "nx": 128, "ny": 128,
         "nz": 128, "dx": 0.2, "eta": 0.35, "mixed": False, "veff": False, "vext": True,
         "fcc": False},
        # a solute in a fine 256^3 box, the largest single evaluation
        {"name": "solute_256", "do": "energy_grad", "hs": "wb", "nx": 256, "ny": 256, "nz": 256,
         "dx": 0.1, "eta": 0.35, "mixed": False, "veff": False, "vext": False, "fcc": False},
        # the mixed form's evaluation, the inner call of a fast solve
        {"name": "mixed_128", "do": "energy_grad", "hs": "wb", "nx": 128, "ny": 128, "nz": 128,
         "dx": 0.2, "eta": 0.3, "mixed": True, "veff": False, "vext": False, "fcc": False},
        # HardSpheres() of the reference (tensor third term) on a ragged box
        {"name": "tensor_ragged", "do": "energy_grad", "hs": "wbt", "nx": 96, "ny": 80, "nz": 100,
         "dx": 0.2, "eta": 0.3, "mixed": False, "veff": False, "vext": False, "fcc": False},
        # liquid water around a hard solute
        {"name": "water_96", "do": "energy_grad", "hs": "water", "nx": 96, "ny": 96, "nz": 96,
         "dx": 0.25, "eta": 0.0, "mixed": False, "veff": False, "vext": False, "fcc": False},
        # a whole slit minimisation in FP64, many evaluations in a row
        {"name": "solve_slit_64", "do": "solve", "n": 64, "dx": 0.2, "eta": 0.3, "width": 6.4,
         "solutes": 0, "mixed": False},
        # the fast path to a converged profile: network, then mixed solve
        {"name": "warm_solve_128", "do": "warm_solve", "n": 128, "dx": 0.2, "eta": 0.3,
         "width": 7.0, "solutes": 2},
        # a small parameter sweep over uneven grids in one call
        {"name": "batch_12", "do": "batch", "count": 12, "largest": 96, "dx": 0.2},
        # the network alone: inference at the size it was trained for
        {"name": "network_128", "do": "network", "n": 128, "channels": 16, "modes": 12,
         "layers": 4, "grad": False},
        # one training sample: loss and parameter gradient
        {"name": "network_grad_96", "do": "network", "n": 96, "channels": 16, "modes": 12,
         "layers": 4, "grad": True},
    ]


def _smooth(rng, lo, hi):
    """A grid edge in [lo, hi] with prime factors up to 13, spread over the logarithm."""
    def ok(n):
        for p in (2, 3, 5, 7, 11, 13):
            while n % p == 0:
                n //= p
        return n == 1
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if lo <= n <= hi and ok(n):
            return n


def draw(rng):
    do = rng.choice(["energy_grad"] * 7 + ["solve"] * 2 + ["warm_solve", "batch"] + ["network"] * 2)
    if do == "energy_grad":
        hs = rng.choice(["wb", "wb", "wb", "rf", "m2", "wbt", "tz", "water"])
        hi = 112 if hs in ("wbt", "tz", "water") else 224
        n = _smooth(rng, 24, hi)
        shape = rng.choice(["cube", "ragged", "two"])
        if shape == "cube":
            nx = ny = nz = n
        elif shape == "ragged":
            nx, ny, nz = (_smooth(rng, max(20, n // 2), n) for _ in range(3))
        else:  # powers of two
            nx = ny = nz = 1 << min(7, max(5, int(round(math.log2(n)))))
        fused = hs in ("wb", "rf", "m2")
        return {"do": do, "hs": hs, "nx": nx, "ny": ny, "nz": nz,
                "dx": 0.25 if hs == "water" else round(rng.uniform(0.1, 0.25), 3),
                "eta": round(rng.uniform(0.1, 0.4), 3), "mixed": fused and rng.random() < 0.35,
                "veff": False, "vext": fused and rng.random() < 0.3,
                "fcc": hs == "wb" and rng.random() < 0.25} | (
                    {"veff": True, "mixed": False} if hs == "wb" and rng.random() < 0.25 else {})
    if do in ("solve", "warm_solve"):
        n = 128 if do == "warm_solve" else rng.choice([32, 36, 40, 48, 56, 60, 64, 72])
        c = {"do": do, "n": n, "dx": 0.2, "eta": round(rng.uniform(0.12, 0.38), 3),
             "width": round(rng.uniform(0.3, 0.65) * n * 0.2, 2), "solutes": rng.randint(0, 3)}
        return c if do == "warm_solve" else c | {"mixed": rng.random() < 0.5}
    if do == "batch":
        return {"do": do, "count": rng.randint(4, 14), "largest": rng.choice([48, 64, 96]),
                "dx": 0.2}
    n = 4 * rng.randint(8, 30)
    return {"do": do, "n": n, "channels": rng.choice([4, 8, 16]),
            "modes": rng.randint(4, min(12, n // 4)), "layers": rng.randint(2, 4),
            "grad": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# Inputs

HS = {"wb": _lib.HS_WB_NOTENSOR, "rf": _lib.HS_RF, "m2": _lib.HS_WB_MARK2,
      "wbt": _lib.HS_WB_TENSOR, "tz": _lib.HS_TARAZONA, "water": _lib.HS_WB_NOTENSOR}


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _noise(shape, dx, seed, sigma=0.4):
    """Gaussian noise smoothed over sigma, unit RMS."""
    xi = torch.randn(shape, generator=_gen(seed), device=DEV, dtype=torch.float64)
    k = [2 * math.pi * torch.fft.fftfreq(n, dx, device=DEV, dtype=torch.float64) for n in shape]
    kz = 2 * math.pi * torch.fft.rfftfreq(shape[2], dx, device=DEV, dtype=torch.float64)
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + kz[None, None, :] ** 2
    xi = torch.fft.irfftn(torch.fft.rfftn(xi) * torch.exp(-0.5 * k2 * sigma * sigma), s=shape)
    return xi / xi.square().mean().sqrt()


def _free(shape, dx, width, solutes, seed):
    """1 where the fluid may be: 0 < z < width, outside `solutes` spheres placed by the seed."""
    c = [torch.arange(n, device=DEV, dtype=torch.float64) * dx for n in shape]
    free = ((c[2] > 1e-12) & (c[2] < width - 1e-12)).expand(shape).clone()
    rng = np.random.default_rng(seed)
    box = [n * dx for n in shape]
    for _ in range(solutes):
        at = [rng.uniform(0, box[0]), rng.uniform(0, box[1]), rng.uniform(0, width)]
        radius = rng.uniform(0.08, 0.16) * min(box)
        d = [torch.minimum((x - a).abs(), b - (x - a).abs()) for x, a, b in zip(c, at, box)]
        r2 = d[0][:, None, None] ** 2 + d[1][None, :, None] ** 2 + d[2][None, None, :] ** 2
        free &= r2 > radius * radius
    return free.double()


def _nq(kT):
    x = 18.01528 * 1822.8885 * kT / (2 * math.pi)
    return x * math.sqrt(x)


def _bulk_mu(hs, R, kT, nb):
    """The chemical-potential coefficient that makes nb the bulk density."""
    n = torch.tensor(nb, dtype=torch.float64, requires_grad=True)
    zero = torch.zeros((), dtype=torch.float64)
    w = [n * 4 * math.pi / 3 * R ** 3, n * 4 * math.pi * R * R, zero, zero, zero] + [zero] * 6
    (d,) = torch.autograd.grad(sum(_phi(hs, R, w)), n)
    return -(kT * float(d) + kT * math.log(nb / _nq(kT)))


def _fields(case, seed):
    """The inputs of an energy_grad case: lattice, R, kT, mu, density n, mask, V."""
    shape, dx, hs = (case["nx"], case["ny"], case["nz"]), case["dx"], case["hs"]
    if case["fcc"]:
        a = [n * dx / math.sqrt(2) for n in shape]
        lat = np.array([[0, a[0], a[0]], [a[1], 0, a[1]], [a[2], a[2], 0.0]])
        if np.linalg.det(lat) < 0:
            lat = lat[::-1].copy()
    else:
        lat = np.diag([n * dx for n in shape])
    if hs == "water":
        R, kT, nb, mu, floor = WATER_R, WATER_KT, WATER_N, WATER_MU, 1e-5
        c = [(torch.arange(n, device=DEV, dtype=torch.float64) - n / 2) * dx for n in shape]
        r2 = c[0][:, None, None] ** 2 + c[1][None, :, None] ** 2 + c[2][None, None, :] ** 2
        mask = (r2 > (0.25 * min(shape) * dx) ** 2).double()
        amp = 0.02
    else:
        R, kT, floor, amp = 1.0, 1.0, 0.0, 0.05
        nb = case["eta"] / (4 * math.pi / 3)
        mu = _bulk_mu(hs, R, kT, nb)
        mask = _free(shape, dx, 0.6 * shape[2] * dx, 1, seed)
        if case["veff"] or hs in ("wbt", "tz"):
            floor = 1e-4
    n = nb * (1 + amp * _noise(shape, dx, seed).clamp(-4, 4)) * mask + floor * nb * (1 - mask)
    V = 0.3 * _noise(shape, dx, seed + 7919, 0.8) if case["vext"] else None
    return lat, R, kT, mu, n.contiguous(), mask.contiguous(), V


class State:
    """What the program keeps; gives the library's objects back when it goes."""

    def __init__(self, case):
        self.case, self.L, self.closers = case, _lib.load(), []

    def make(self, create, destroy, *args):
        h = ctypes.c_void_p()
        _lib.check(create(*args, ctypes.byref(h)))
        self.closers.append(lambda: destroy(h))
        return h

    def __del__(self):
        while self.closers:
            self.closers.pop()()


def _functional(s, lat, shape, R, kT, mu, terms, mixed, hs, mask=None, V=None, saft=None):
    L, ctx = s.L, default_context()
    lat9 = np.ascontiguousarray(np.asarray(lat, dtype=np.float64).reshape(9))
    s.grid = s.make(L.deft_grid_create, L.deft_grid_destroy, ctx.handle, lat9.ctypes.data, *shape)
    p = _lib.FmtParams(R, kT, mu, terms, int(mixed), hs)
    f = s.make(L.deft_fmt_create, L.deft_fmt_destroy, s.grid, ctypes.byref(p))
    torch.cuda.synchronize()
    if mask is not None:
        _lib.check(L.deft_fmt_set_mask(f, mask.data_ptr(), 1))
    if V is not None:
        _lib.check(L.deft_fmt_set_vext(f, V.data_ptr(), 1))
    if saft is not None:
        sp = np.array(saft)
        _lib.check(L.deft_fmt_set_saft(f, sp.ctypes.data))
    ctx.sync()
    return f


def _problem(case, seed):
    """Geometry, mask and bulk start of a hard-sphere solve."""
    shape, dx = (case["n"],) * 3, case["dx"]
    nb = case["eta"] / (4 * math.pi / 3)
    mask = _free(shape, dx, case["width"], case["solutes"], seed)
    n0 = nb * mask
    if case["do"] == "solve":
        n0 = n0 * (1 + 0.05 * _noise(shape, dx, seed).clamp(-4, 4))
    return shape, np.diag([n * dx for n in shape]), nb, _bulk_mu("wb", 1.0, 1.0, nb), mask, n0


HARD = _lib.TERM_HS | _lib.TERM_IDEAL | _lib.TERM_MU | _lib.TERM_MASK
# |grad F| of the solves: tight enough that the profile is fixed to about 1e-10
GTOL = 1e-11


class _Problem:
    """One problem of a batch, as solve_batch takes it."""


def _net_inputs(case, seed):
    n = case["n"]
    dx = 25.6 / n
    mask = _free((n,) * 3, dx, 0.5 * n * dx, 2, seed)
    target = mask * (1 + 0.2 * _noise((n,) * 3, dx, seed).clamp(-4, 4))
    return mask.float().contiguous(), target.float().contiguous()


def _net_params(net_size, seed):
    """Parameters of the size of a trained network's: the initial ones are
    small random numbers too."""
    g = np.random.default_rng(seed)
    return (0.05 * g.standard_normal(net_size, dtype=np.float32)).astype(np.float32)


def _net_layout(case):
    C, m, layers = case["channels"], case["modes"], case["layers"]
    at, o = {}, 0
    K = 4 * m * m * m
    sizes = [("P", 2 * C), ("p", C)]
    for l in range(layers):
        sizes += [("W%d" % l, 2 * C * C * K), ("Wp%d" % l, C * C), ("b%d" % l, C)]
    sizes += [("Q1", C * C), ("q1", C), ("Q2", C), ("q2", 1)]
    for name, n in sizes:
        at[name] = (o, n)
        o += n
    return at, o


def _net_weights(case, seed):
    at, size = _net_layout(case)
    p = _net_params(size, seed)
    for l in range(case["layers"]):  # the pointwise maps keep the signal's size
        o, n = at["Wp%d" % l]
        p[o:o + n] *= 5.0
        o, n = at["W%d" % l]
        p[o:o + n] *= 0.4
    for name in ("P", "Q1", "Q2"):
        o, n = at[name]
        p[o:o + n] *= 10.0
    return p


def prepare(case, seed):
    s = State(case)
    L = s.L
    if case["do"] == "energy_grad":
        lat, R, kT, mu, n, s.mask, s.V = _fields(case, seed)
        terms = _lib.TERM_HS | _lib.TERM_IDEAL | _lib.TERM_MU | _lib.TERM_MASK
        terms |= _lib.TERM_VEXT if s.V is not None else 0
        terms |= _lib.TERM_VEFF if case["veff"] else 0
        terms |= _lib.TERM_SAFT if case["hs"] == "water" else 0
        s.x = -kT * torch.log(n) if case["veff"] else n
        s.g, s.pg = torch.empty_like(n), torch.empty_like(n) if case["veff"] else None
        s.f = _functional(s, lat, n.shape, R, kT, mu, terms, case["mixed"], HS[case["hs"]], s.mask,
                          s.V, WATER if case["hs"] == "water" else None)
    elif case["do"] in ("solve", "warm_solve"):
        shape, lat, s.nb, mu, s.mask, s.n0 = _problem(case, seed)
        mixed = case["do"] == "warm_solve" or case["mixed"]
        s.f = _functional(s, lat, shape, 1.0, 1.0, mu, HARD, mixed, 0, s.mask)
        structure = mixed and case["n"] in (32, 64, 128, 256)
        s.p = _lib.CgParams(_lib.LS_SECANT, GTOL, 20000, 1.0, 0.0, 0.0,
                            _lib.PC_STRUCTURE if structure else _lib.PC_DENSITY)
        s.cg = s.make(L.deft_cg_create, L.deft_cg_destroy, s.f, ctypes.byref(s.p))
        s.st = _lib.CgStatus()
        s.out = torch.empty_like(s.n0)
        if case["do"] == "warm_solve":
            s.net = FourierOperator.load(WEIGHTS)
            s.closers.append(s.net.close)
            s.start = torch.empty_like(s.n0)
    elif case["do"] == "batch":
        rng = np.random.default_rng(seed)
        s.problems = []
        edges = [v for v in (96, 64, 48, 32) if v <= case["largest"]]
        for k in range(case["count"]):
            n = edges[k % len(edges)]
            width = min(float(rng.uniform(3.0, 10.0)), 0.7 * n * case["dx"])
            one = {"do": "solve", "n": n, "dx": case["dx"], "eta": float(rng.uniform(0.05, 0.4)),
                   "width": width, "solutes": 0}
            p = _Problem()
            p.shape, p.lat, _, p.mu, mask, n0 = _problem(one, seed * 100 + k)
            p.R, p.kT, p.mask, p.n0 = 1.0, 1.0, mask.cpu().numpy(), n0.cpu().numpy()
            s.problems.append(p)
    else:
        s.mask, s.target = _net_inputs(case, seed)
        s.net = FourierOperator(case["n"], case["channels"], case["modes"], case["layers"])
        s.closers.append(s.net.close)
        s.net.set_params(_net_weights(case, seed))
        s.eta, s.y = 0.1 + 0.3 * ((seed * 0.6180339887) % 1), torch.empty_like(s.mask)
        s.grad = np.empty(s.net.nparam, dtype=np.float32) if case["grad"] else None
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# One pass

def run(s):
    L, case = s.L, s.case
    if case["do"] == "energy_grad":
        E = ctypes.c_double()
        if s.pg is not None:
            _lib.check(L.deft_fmt_energy_grad_pgrad(s.f, s.x.data_ptr(), 1, ctypes.addressof(E),
                                                    s.g.data_ptr(), s.pg.data_ptr(), None))
            return {"energy": E.value, "grad": s.g, "pgrad": s.pg}
        _lib.check(L.deft_fmt_energy_grad(s.f, s.x.data_ptr(), 1, ctypes.addressof(E),
                                          s.g.data_ptr(), None))
        if case["mixed"]:  # FP32 transforms: the program keeps what they carry
            return {"energy": np.float32(E.value), "grad": s.g.float()}
        return {"energy": E.value, "grad": s.g}
    if case["do"] in ("solve", "warm_solve"):
        start = s.n0
        if case["do"] == "warm_solve":
            start = s.start
            _, _, gb = s.net.initial_density(s.f, s.mask.data_ptr(), case["eta"], s.nb,
                                             start.data_ptr(), bulk_gnorm=True)
            s.p.refine_abs = 3e-6 * gb
            _lib.check(L.deft_cg_set_params(s.cg, ctypes.byref(s.p)))
        _lib.check(L.deft_cg_set_x(s.cg, start.data_ptr(), 1))
        _lib.check(L.deft_cg_solve(s.cg, ctypes.byref(s.st)))
        _lib.check(L.deft_cg_get_x(s.cg, s.out.data_ptr(), 1))
        return {"energy": s.st.energy, "profile": s.out}
    if case["do"] == "batch":
        code, st, profiles = solve_batch(s.problems, gtol=GTOL, preconditioned=_lib.PC_STRUCTURE)
        _lib.check(code)
        return {"energies": [v.energy for v in st], "profiles": profiles}
    loss = ctypes.c_float()
    if s.grad is None:
        _lib.check(L.deft_fno_eval(s.net.h, s.mask.data_ptr(), s.eta, None, 1, s.y.data_ptr(),
                                   None, None))
        return {"y": s.y}
    _lib.check(L.deft_fno_eval(s.net.h, s.mask.data_ptr(), s.eta, s.target.data_ptr(), 1,
                               s.y.data_ptr(), ctypes.addressof(loss), s.grad.ctypes.data))
    return {"y": s.y, "loss": np.float32(loss.value), "grad": s.grad}


# ---------------------------------------------------------------------------
# What a pass cannot do without

def work(case):
    if case["do"] == "network":
        C, layers, n3 = case["channels"], case["layers"], case["n"] ** 3
        size = _net_layout(case)[1]
        # transforms cut to the kept modes, the mode mixing, the pointwise maps
        per = 2 * n3 * C * C + 8 * C * C * 4 * case["modes"] ** 3 + 5 * C * n3 * math.log2(n3)
        flops = layers * per + n3 * (2 * C * C + 6 * C)
        if case["grad"]:  # each product once more for either of its factors
            return {"bytes": 4.0 * (3 * n3) + 6.0 * size, "flops": 3 * flops}
        return {"bytes": 4.0 * (2 * n3) + 2.0 * size, "flops": flops}
    if case["do"] == "energy_grad":
        n3 = case["nx"] * case["ny"] * case["nz"]
        fields = 3 + bool(case["vext"]) + bool(case["veff"])
        return {"bytes": 8.0 * fields * n3, "flops": _eval_flops(case["hs"], n3)}
    if case["do"] == "batch":
        # about 25 evaluations or products of each problem
        edges = [v for v in (96, 64, 48, 32) if v <= case["largest"]]
        n3 = sum(edges[k % len(edges)] ** 3 for k in range(case["count"]))
        return {"bytes": 3 * 8.0 * n3, "flops": 25 * _eval_flops("wb", n3)}
    n3 = case["n"] ** 3
    # a converged solve takes at least some twenty evaluations of its size
    flops = 20 * _eval_flops("wb", n3)
    return {"bytes": 3 * 8.0 * n3, "flops": flops}


def _eval_flops(hs, n3):
    transforms = {"wbt": 24, "tz": 24, "water": 40}.get(hs, 12)
    return transforms * 2.5 * n3 * math.log2(n3) + 150 * n3


# ---------------------------------------------------------------------------
# The same in 64 bits, in plain torch

def _S(e):
    """(e + (1-e)^2 ln(1-e)) / e^2, by its series where that cancels."""
    small = e.abs() < 0.1
    x = torch.where(small, torch.full_like(e, 0.5), e)
    closed = (x + (1 - x) ** 2 * torch.log1p(-x)) / x ** 2
    y = torch.where(small, e, torch.zeros_like(e))
    series = torch.zeros_like(e)
    for j in range(24, 0, -1):
        series = (series + 2.0 / (j * (j + 1) * (j + 2))) * y
    return torch.where(small, 1.5 - series, closed)


def _dS(e):
    small = e.abs() < 0.1
    x = torch.where(small, torch.full_like(e, 0.5), e)
    l = torch.log1p(-x)
    closed = (x - 2 * (1 - x) * l - 2 * (x + (1 - x) ** 2 * l) / x) / x ** 2
    y = torch.where(small, e, torch.zeros_like(e))
    series = torch.zeros_like(e)
    for j in range(24, 0, -1):
        series = series * y + 2.0 / ((j + 1) * (j + 2))
    return torch.where(small, -series, closed)


def _m2(e):
    """P2, P3 of White Bear mark II."""
    small = e.abs() < 0.2
    x = torch.where(small, torch.full_like(e, 0.5), e)
    l = torch.log1p(-x)
    p2 = 1 + (6 - 3 * x + 6 * (1 - x) * l / x) / 9
    p3 = 1 - (6 - 9 * x + 6 * x * x + 6 * (1 - x) ** 2 * l / x) / (9 * x)
    y = torch.where(small, e, torch.zeros_like(e))
    s2, s3 = torch.zeros_like(e), torch.zeros_like(e)
    for k in range(32, 1, -1):
        s2 = s2 * y + 1.0 / (k * (k + 1))
        if k > 2:
            s3 = s3 * y + 1.0 / ((k - 1) * k * (k + 1))
    return (torch.where(small, 1 + 2.0 / 3 * y * y * s2, p2),
            torch.where(small, 1 - 4.0 / 9 * y + 4.0 / 3 * y * y * s3, p3))


def _phi(hs, R, w):
    """phi1, phi2, phi3 per kT of the weighted densities n3, n2, vx, vy, vz (and the tensor's
    xx, yy, zz, xy, yz, zx)."""
    n3, n2, vx, vy, vz = w[:5]
    u, l = 1 / (1 - n3), torch.log1p(-n3)
    v2 = vx * vx + vy * vy + vz * vz
    third = n2 ** 3 - 3 * n2 * v2
    f2 = u
    if hs == "m2":
        P2, P3 = _m2(n3)
        f2, f3 = P2 * u, P3 * u * u / (24 * math.pi)
    elif hs in ("rf", "tz"):
        f3 = u * u / (24 * math.pi)
    else:
        f3 = _S(n3) * u * u / (36 * math.pi)
    if hs in ("wbt", "tz"):
        xx, yy, zz, xy, yz, zx = w[5:11]
        T = [[xx, xy, zx], [xy, yy, yz], [zx, yz, zz]]
        v = [vx, vy, vz]
        vTv = sum(v[i] * T[i][j] * v[j] for i in range(3) for j in range(3))
        tr3 = sum(T[i][j] * T[j][k] * T[k][i] for i in range(3) for j in range(3) for k in range(3))
        third = third + 9 * (vTv - 0.5 * tr3)
    return (-n2 * l / (4 * math.pi * R * R), (n2 * n2 - v2) * f2 / (4 * math.pi * R), third * f3)


class _Space:
    """Convolutions with the analytic weights on one grid."""

    def __init__(self, lat, shape):
        self.shape = tuple(shape)
        B = 2 * math.pi * np.linalg.inv(np.asarray(lat, dtype=np.float64)).T  # rows: reciprocal
        m = []
        for i, n in enumerate(shape):
            v = np.arange(n if i < 2 else n // 2 + 1)
            if i < 2:
                v = np.where(v > n // 2, v - n, v)
            m.append(torch.tensor(v, device=DEV, dtype=torch.float64))
        self.k = [B[0, c] * m[0][:, None, None] + B[1, c] * m[1][None, :, None]
                  + B[2, c] * m[2][None, None, :] for c in range(3)]
        self.k2 = sum(k * k for k in self.k)
        self.zero = self.k2 == 0
        self.k2 = torch.where(self.zero, torch.ones_like(self.k2), self.k2)
        self.kk = self.k2.sqrt()
        self.dV = abs(np.linalg.det(lat)) / np.prod(self.shape)
        self.smear = torch.exp(-6 * self.k2 * self.dV ** (2.0 / 3))

    def at0(self, w, value):
        return torch.where(self.zero, torch.full_like(w, value), w)

    def step(self, R):
        x = self.kk * R
        return self.at0(self.smear * 4 * math.pi * (torch.sin(x) - x * torch.cos(x)) / self.kk ** 3,
                        4 * math.pi / 3 * R ** 3)

    def shell(self, R):
        return self.at0(self.smear * 4 * math.pi * R * torch.sin(self.kk * R) / self.kk,
                        4 * math.pi * R * R)

    def shell_prime(self, R):  # with its sign turned
        x = self.kk * R
        return self.at0(self.smear * 4 * math.pi * (torch.sin(x) / self.kk + R * torch.cos(x)),
                        8 * math.pi * R)

    def vshell(self, c, R):  # the imaginary part
        x = self.kk * R
        return self.at0(self.smear * 4 * math.pi * self.k[c] / self.k2
                        * (R * torch.cos(x) - torch.sin(x) / self.kk), 0.0)

    def vshell_prime(self, c, R):
        return self.at0(self.smear * 4 * math.pi * R * self.k[c] / self.kk
                        * torch.sin(self.kk * R), 0.0)

    def tensor(self, a, R):
        x = self.kk * R
        s, c, x2 = torch.sin(x), torch.cos(x), x * x
        if a < 3:
            q = self.k[a] ** 2 / self.k2
            w = self.smear * 4 * math.pi * R * R * (
                s / x * (-1.0 / 3 + q - 3 * q / x2 + 1 / x2) + c / x2 * (3 * q - 1))
        else:
            i, j = a - 3, (a - 2) % 3
            w = -self.smear * 4 * math.pi * self.k[i] * self.k[j] / self.k2 ** 2 * (
                (3 - x2) * s / x - 3 * c)
        return self.at0(w, 0.0)

    def back(self, F):
        return torch.fft.irfftn(F, s=self.shape)

    def weighted(self, F, R, tensor=False):
        w = [self.back(F * self.step(R)), self.back(F * self.shell(R))]
        w += [self.back(F * (1j * self.vshell(c, R))) for c in range(3)]
        if tensor:
            w += [self.back(F * self.tensor(a, R)) for a in range(6)]
        return w


def _water(sp, F, n, w, R, kT):
    """Association and dispersion free-energy densities."""
    eps_a, kap, eps_d, lam, ls = WATER
    n3, n2, v = w[0], w[1], w[2:5]
    v2 = sum(x * x for x in v)
    c1 = 1 / (4 * math.pi * R)
    c0 = c1 / R
    u = 1 / (1 - n3)
    S = _S(n3)
    f3 = S * u * u / (36 * math.pi)
    f3p = (_dS(n3) + 2 * S * u) * u * u / (36 * math.pi)
    q, t3 = n2 * n2 - v2, n2 * (n2 * n2 - 3 * v2)
    d0, d1 = -torch.log1p(-n3), n2 * u
    d2, d3 = c1 * n2 * u + 3 * q * f3, c0 * n2 * u + c1 * q * u * u + t3 * f3p
    d1v, d2v = -u, -c1 * u - 6 * n2 * f3
    A = torch.fft.rfftn(d3 - 2 * c0 / R * d0 - c0 * d1) * sp.shell(R)
    A = A + torch.fft.rfftn(d2 + c1 * d1 + c0 * d0) * sp.shell_prime(R)
    for c in range(3):
        A = A + torch.fft.rfftn(v[c] * c0 * d1v) * (1j * sp.vshell(c, R))
        A = A + torch.fft.rfftn(v[c] * (c1 * d1v + d2v)) * (1j * sp.vshell_prime(c, R))
    A = sp.back(A)
    D = sp.back(F * sp.shell(2 * R))
    s = 2 * ls * lam * R
    k2 = torch.where(sp.zero, torch.zeros_like(sp.k2), sp.k2)
    eta = 4 * math.pi / 3 * R ** 3 * sp.back(F * torch.exp(-0.5 * k2 * s * s))
    c = (2.25855 - 1.50349 * lam + 0.249434 * lam * lam,
         -0.669270 + 1.40049 * lam - 0.827739 * lam * lam,
         10.1576 - 15.0427 * lam + 5.30827 * lam * lam)
    cl = (-1.50349 + 2 * 0.249434 * lam, 1.40049 - 2 * 0.827739 * lam,
          -15.0427 + 2 * 5.30827 * lam)
    x = (c[0] + c[1] * eta + c[2] * eta ** 2) * eta
    xe = c[0] + 2 * c[1] * eta + 3 * c[2] * eta ** 2
    xl = (cl[0] + cl[1] * eta + cl[2] * eta ** 2) * eta
    g, g1 = (1 - x / 2) / (1 - x) ** 3, (2.5 - x) / (1 - x) ** 4
    L3 = lam ** 3 - 1
    a1 = -4 * eps_d * L3 * eta * g
    a1e = -4 * eps_d * L3 * (g + eta * g1 * xe)
    a1l = -4 * eps_d * eta * (3 * lam * lam * g + L3 * g1 * xl)
    a2 = 0.5 * (1 - eta) ** 4 / (1 + 2 * eta) ** 2 * eps_d * eta * a1e
    gsw = A / D + (a1e - lam / (3 * eta) * a1l) / (4 * kT)
    y = D / (16 * math.pi * R * R) * gsw * kap * (math.exp(eps_a / kT) - 1)
    X = (torch.sqrt(1 + 8 * y) - 1) / (4 * y)
    return 4 * kT * n * (torch.log(X) - X / 2 + 0.5) + n * a1 + n * a2 / kT


def _energy(sp, hs, R, kT, mu, n, V):
    F = torch.fft.rfftn(n)
    w = sp.weighted(F, R, hs in ("wbt", "tz"))
    there = n > 0
    ln = torch.log(torch.where(there, n, torch.ones_like(n)) / _nq(kT))
    e = kT * sum(_phi("wb" if hs == "water" else hs, R, w))
    e = e + torch.where(there, kT * n * (ln - 1), torch.zeros_like(n)) + mu * n
    if hs == "water":
        e = e + _water(sp, F, n, w, R, kT)
    if V is not None:
        e = e + V * n
    return sp.dV * e.sum()


def _energy_grad(sp, hs, R, kT, mu, n, mask, V):
    n = n.detach().requires_grad_(True)
    E = _energy(sp, hs, R, kT, mu, n, V)
    (g,) = torch.autograd.grad(E, n)
    return E.item(), torch.where(mask == 0, torch.zeros_like(g), g * mask)


def _minimise(sp, mu, n, mask, gtol):
    """Conjugate gradient (Polak-Ribiere, preconditioned with n / dV) with a
    secant search on the slope; None if it does not get there."""
    dot = lambda a, b: float((a * b).sum())  # noqa: E731
    E, g = _energy_grad(sp, "wb", 1.0, 1.0, mu, n, mask, None)
    z, d, rz, step = n * g / sp.dV, None, 0.0, 0.5
    for _ in range(400):
        if math.sqrt(dot(g, g)) < gtol:
            return E, n
        new = dot(z, g)
        d = -z if d is None else d * max(0.0, (new - dot(z, old)) / rz) - z
        if dot(d, g) >= 0:
            d = -z
        rz, old, s0 = new, g, dot(d, g)
        a0, sa, a = 0.0, s0, step
        for _ in range(12):
            at = n + a * d
            if float(at.min()) < 0:
                a = 0.5 * (a0 + a)
                continue
            E, g = _energy_grad(sp, "wb", 1.0, 1.0, mu, at, mask, None)
            s = dot(g, d)
            if abs(s) <= 0.3 * abs(s0):
                break
            to = a - s * (a - a0) / (s - sa) if s != sa else 2 * a
            if s < 0 and to <= a:
                to = 2 * a
            a0, sa, a = a, s, min(max(to, 0.05 * a), 4 * a)
        n, step = at, a
        z = n * g / sp.dV
    return None


def _network(case, p, mask, target, eta):
    at, _ = _net_layout(case)
    C, m, N = case["channels"], case["modes"], case["n"]
    get = lambda name: p[at[name][0]:at[name][0] + at[name][1]]  # noqa: E731
    h = get("P").view(C, 2)[:, 0, None, None, None] * mask
    h = h + (get("P").view(C, 2)[:, 1] * eta + get("p"))[:, None, None, None]
    keep = torch.tensor(list(range(m)) + list(range(N - m, N)), device=DEV)
    for l in range(case["layers"]):
        W = torch.view_as_complex(get("W%d" % l).view(C, C, 2 * m, 2 * m, m, 2))
        F = torch.fft.rfftn(h, dim=(1, 2, 3))[..., :m].index_select(1, keep).index_select(2, keep)
        U = torch.einsum("ioabc,iabc->oabc", W, F)
        G = torch.zeros((C, N, 2 * m, m), dtype=U.dtype, device=DEV).index_add(1, keep, U)
        G = torch.zeros((C, N, N, m), dtype=U.dtype, device=DEV).index_add(2, keep, G)
        G = torch.nn.functional.pad(G, (0, N // 2 + 1 - m))
        h = torch.fft.irfftn(G, s=(N, N, N), dim=(1, 2, 3)) + get("b%d" % l)[:, None, None, None] \
            + torch.einsum("oi,ixyz->oxyz", get("Wp%d" % l).view(C, C), h)
        if l < case["layers"] - 1:
            h = torch.nn.functional.gelu(h)
    a = torch.einsum("ci,ixyz->cxyz", get("Q1").view(C, C), h) + get("q1")[:, None, None, None]
    y = torch.einsum("c,cxyz->xyz", get("Q2"), torch.nn.functional.gelu(a)) + get("q2")
    return y, (mask * (y - target) ** 2).sum() / mask.sum()


def exact(case, seed):
    if case["do"] == "energy_grad":
        lat, R, kT, mu, n, mask, V = _fields(case, seed)
        sp = _Space(lat, n.shape)
        x = -kT * torch.log(n) if case["veff"] else None
        n = torch.exp(-x / kT) if case["veff"] else n
        E, g = _energy_grad(sp, case["hs"], R, kT, mu, n, mask, V)
        if case["veff"]:
            return {"energy": E, "grad": -n * g / kT, "pgrad": g / (x - kT)}
        return {"energy": E, "grad": g}
    if case["do"] in ("solve", "warm_solve"):
        shape, lat, _, mu, mask, n0 = _problem(case, seed)
        got = _minimise(_Space(lat, shape), mu, n0, mask, 0.3 * GTOL)
        return got and {"energy": got[0], "profile": got[1]}
    if case["do"] == "batch":  # a dozen such minimisations take too long
        return None
    mask, target = _net_inputs(case, seed)
    p = torch.tensor(_net_weights(case, seed), device=DEV).bfloat16().double()
    p.requires_grad_(case["grad"])
    eta = float(np.float32(0.1 + 0.3 * ((seed * 0.6180339887) % 1)))
    y, loss = _network(case, p, mask.double(), target.double(), eta)
    if not case["grad"]:
        return {"y": y}
    loss.backward()
    return {"y": y.detach(), "loss": loss.item(), "grad": p.grad.detach()}
