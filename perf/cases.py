"""The evaluation pass as its users run it, case by case.

Each case is one call, or one step, of the public interface over a body set:

  solve     LaplaceFMM.solve(): bodies in host memory, set-up and pass (the
            reference driver's own call)
  evaluate  LaplaceFMM.evaluate(q): a set-up kept, charges and results in host
            memory
  forward   LaplaceFMM.forward_device(): a set-up kept, charges and results in
            device memory
  adjoint   forward_device() then adjoint_device(): one forward and backward
            step of a differentiable program
  step      setup_device() then forward_device(): a time step in which the
            bodies have moved

The listed sizes are those of the named configurations of this repository
(8192 uniform bodies at P = 6; 2^20 at P = 8, and at P = 6 with small leaves,
the fastest setting within 1e-5; 2^22 bodies in 64 blobs and the 200^3 jittered
lattice at P = 10), the reference's default run (1000 bodies, P = 4, ncrit = 16)
and odd sizes between them.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    name = "exafmm_rd_b200"
    if name not in sys.modules:
        d = os.path.join(_ROOT, "exafmm-rd_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _case(name, call, bodies, n, P, ncrit, images, mixed, dipole=0, cycle=1.0):
    c = dict(call=call, bodies=bodies, n=n, P=P, ncrit=ncrit, images=images, mixed=mixed, dipole=dipole, cycle=cycle)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the reference's default run: the smallest call, host set-up and launches
        _case("solve_1k_p4_f64", "solve", "uniform", 1000, 4, 16, 0, False, dipole=1, cycle=2 * math.pi),
        # the small periodic configuration, as one of many passes with new charges
        _case("forward_8k_p6_f64", "forward", "uniform", 8192, 6, 64, 3, False),
        # a gradient step on a small clustered set in free space
        _case("adjoint_30k_p5_mixed", "adjoint", "blobs", 30011, 5, 48, 0, True),
        # one time step of a moving system: octree, lists and pass
        _case("step_100k_p6_mixed", "step", "uniform", 100003, 6, 64, 2, True),
        # FP64 field of a mid-sized clustered set in free space
        _case("forward_blobs_150k_p7_f64", "forward", "blobs", 150001, 7, 100, 0, False),
        # a program whose charges and results live in host memory
        _case("evaluate_200k_p6_mixed", "evaluate", "uniform", 200003, 6, 64, 1, True, dipole=2),
        # 2^20 bodies at the fastest setting within 1e-5
        _case("forward_1m_p6_mixed", "forward", "uniform", 1 << 20, 6, 64, 3, True),
        # the headline configuration, in both forms
        _case("forward_1m_p8_mixed", "forward", "uniform", 1 << 20, 8, 256, 3, True),
        _case("forward_1m_p8_f64", "forward", "uniform", 1 << 20, 8, 256, 3, False),
        # its differentiable form
        _case("adjoint_1m_p8_mixed", "adjoint", "uniform", 1 << 20, 8, 256, 3, True),
        # the clustered configuration at high order
        _case("forward_blobs_4m_p10_mixed", "forward", "blobs", 1 << 22, 10, 128, 3, True),
        # the ionic lattice, forward and backward: the largest
        _case("adjoint_lattice_8m_p10_mixed", "adjoint", "lattice", 200 ** 3, 10, 256, 4, True),
    ]


def draw(rng):
    while True:
        call = rng.choice(["solve", "evaluate", "forward", "forward", "adjoint", "adjoint", "step"])
        bodies = rng.choice(["uniform", "uniform", "blobs", "lattice"])
        n = int(round(math.exp(rng.uniform(math.log(1000), math.log(4.2e6)))))
        if bodies == "lattice":
            n = max(10, 2 * int(round(n ** (1.0 / 3) / 2))) ** 3
        P = rng.choice([4, 5, 6, 7, 8, 9, 10])
        ncrit = int(round(math.exp(rng.uniform(math.log(32), math.log(400)))))
        c = _case(None, call, bodies, n, P, ncrit, rng.choice([0, 1, 2, 3, 3, 4]), rng.random() < 0.6,
                  dipole=rng.choice([0, 0, 0, 2]), cycle=rng.choice([1.0, 1.0, 2 * math.pi]))
        # no dearer than the listed ones; the M2L spectra of three states fit the card
        if _cost(c) <= 0.6 * _cost(listed()[-1]) and _leaves(c)[0] <= 60000:
            return c


# -- bodies -----------------------------------------------------------------------
def _bodies(case, seed):
    """Positions (n, 3), charges (n) and loss weights (n) on the GPU, FP64."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    n, L = case["n"], case["cycle"]
    kw = dict(generator=g, device="cuda", dtype=torch.float64)
    if case["bodies"] == "uniform":
        x = torch.rand((n, 3), **kw)
        q = torch.rand(n, **kw) * 2 - 1
    elif case["bodies"] == "blobs":
        centre = torch.rand((64, 3), **kw)
        which = torch.randint(0, 64, (n,), generator=g, device="cuda")
        x = torch.remainder(centre[which] + 0.02 * torch.randn((n, 3), **kw), 1.0)
        q = (torch.rand(n, **kw) < 0.5).to(torch.float64) * 2 - 1
    else:  # rock salt, jittered
        m = round(n ** (1.0 / 3))
        k = torch.arange(n, device="cuda")
        ijk = torch.stack([k // (m * m), k // m % m, k % m], 1)
        x = (ijk.to(torch.float64) + 0.5 + 0.2 * torch.rand((n, 3), **kw) - 0.1) / m
        q = 1.0 - 2.0 * (ijk.sum(1) % 2).to(torch.float64)
    q = q - q.mean()
    w = q.clone() if case["bodies"] == "lattice" else torch.randn(n, **kw)  # L = 1/2 sum q phi, or sum w phi
    return (x * L).contiguous(), q, w


def prepare(case, seed):
    pkg = _package()
    x, q, w = _bodies(case, seed)
    torch.cuda.synchronize()
    L = case["cycle"]
    args = pkg.Argument(P=case["P"], ncrit=case["ncrit"], images=case["images"], cycle=L, x=(L / 2, L / 2, L / 2),
                        dipole_correction=case["dipole"], divide_4pi=1, device=0,
                        precision=pkg.FP32_MIXED if case["mixed"] else pkg.FP64)
    s = {"call": case["call"]}
    if case["call"] in ("solve", "evaluate"):
        s["q"] = q.cpu().numpy()
        s["fmm"] = pkg.LaplaceFMM(x.cpu().numpy(), s["q"], args)
        if case["call"] == "evaluate":
            s["fmm"].setup()
            s["fmm"].upload()
        return s
    n = case["n"]
    s["fmm"] = pkg.LaplaceFMM(np.empty((0, 3)), np.empty(0), args)
    s["x"], s["q"], s["w"] = x, q, w
    s["phi"] = torch.empty(n, dtype=torch.float64, device="cuda")
    s["grad"] = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    if case["call"] == "adjoint":
        s["dq"] = torch.empty(n, dtype=torch.float64, device="cuda")
        s["dx"] = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    s["fmm"].setup_device(x.data_ptr(), q.data_ptr(), n)
    return s


def run(s):
    f = s["fmm"]
    if s["call"] == "solve":
        return list(f.solve())
    if s["call"] == "evaluate":
        return list(f.evaluate(s["q"]))
    if s["call"] == "step":
        f.setup_device(s["x"].data_ptr(), s["q"].data_ptr(), len(s["q"]))
    f.forward_device(s["q"].data_ptr(), s["phi"].data_ptr(), s["grad"].data_ptr())
    if s["call"] == "adjoint":
        f.adjoint_device(s["w"].data_ptr(), s["dq"].data_ptr(), s["dx"].data_ptr())
        return [s["phi"], s["grad"], s["dq"], s["dx"]]
    return [s["phi"], s["grad"]]


# -- what a pass cannot do without ------------------------------------------------
def _leaves(case):
    """(leaves, cells above them, mean bodies of a target's neighbouring leaf),
    estimated: a uniform set fills the levels where n / 8^d passes ncrit, a
    clustered one leaves about 0.45 ncrit to a leaf."""
    n, ncrit = case["n"], case["ncrit"]
    if case["bodies"] == "blobs":
        leaves = max(1.0, n / (0.45 * ncrit))
        return leaves, leaves / 6.0, 0.45 * ncrit
    d, leaves, m = 0, 1.0, float(n)
    while m > ncrit:
        d, leaves, m = d + 1, leaves * 8, m / 8
    return leaves, (leaves - 1) / 7, m


def _cost(case):
    """Floating-point operations of one pass, FP64 ones counted twice."""
    n, P = case["n"], case["P"]
    leaves, parents, m = _leaves(case)
    ns = 6 * (P - 1) ** 2 + 2
    nf = (2 * P - 1) ** 2 * P
    pairs = n * min(n, 27 * m)
    far = 31.0 * n * ns + 8.0 * leaves * ns * ns + 4.0 * (leaves + parents) * ns * ns
    m2l = parents * 26 * 27 * 8.0 * nf
    heavy = 1 if case["mixed"] else 2
    passes = 2 if case["call"] == "adjoint" else 1
    return passes * (heavy * 20.0 * pairs + 2 * far + (heavy if P <= 8 else 2) * m2l)


def work(case):
    """Each body's position and charge read once and its results written once;
    20 operations a near pair, 11 and 20 a body and surface point, 2 ns^2 an
    operator application, and 27 complex products (the 2 x 2 x 2 blocks of
    children are Toeplitz) a target parent, direction and frequency."""
    one = dict(case, mixed=True)
    n, P = case["n"], case["P"]
    leaves, parents, m = _leaves(case)
    ns = 6 * (P - 1) ** 2 + 2
    nf = (2 * P - 1) ** 2 * P
    flops = (20.0 * n * min(n, 27 * m) + 31.0 * n * ns + (8.0 * leaves + 4.0 * (leaves + parents)) * ns * ns
             + parents * 26 * 27 * 8.0 * nf)
    nbytes = n * (32 + 32.0)
    if one["call"] == "adjoint":
        flops *= 2
        nbytes += n * (8 + 32.0)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what the outputs move by when the bodies are given in
    another order, so that every sum runs in another order.  Mixed: 6e-7, and
    2e-6 on the jittered lattice, whose fields are small differences of large
    terms.  FP64: 2e-12 at three image levels and nine times that for each one
    more; from P = 9 on the equivalent densities are as ill-conditioned as
    FP64 holds, and two FP64 implementations agree to about 1e-7."""
    if case["mixed"]:
        return {"rel": 8e-6, "max": 1.6e-4} if case["bodies"] == "lattice" else {"rel": 2.5e-6, "max": 2.5e-5}
    return {"rel": 1e-7, "max": 1e-5} if case["P"] >= 9 else {"rel": 1e-10, "max": 4e-9}


# -- 64-bit values ----------------------------------------------------------------
def _direct(x, q):
    """Free-space sums: potential and gradient, FP64."""
    n = len(x)
    phi, grad = torch.empty_like(q), torch.empty_like(x)
    step = max(1, (1 << 26) // n)
    for a in range(0, n, step):
        d = x[a:a + step, None, :] - x[None, :, :]
        r2 = (d * d).sum(2)
        ir = torch.where(r2 > 0, r2, torch.full_like(r2, math.inf)).rsqrt()
        qir = ir * q
        phi[a:a + step] = qir.sum(1)
        grad[a:a + step] = -torch.einsum("ij,ijk->ik", qir * ir * ir, d)
    return phi, grad


def _ewald(x, q, L, ksize=11):
    """Periodic sums of a neutral set, summed in growing cubes: Ewald's sum
    plus the surface term of that order, FP64."""
    n = len(x)
    alpha = ksize / L
    phi, grad = torch.zeros_like(q), torch.zeros_like(x)
    step = max(1, (1 << 26) // n)
    for a in range(0, n, step):
        d = x[a:a + step, None, :] - x[None, :, :]
        d -= L * torch.round(d / L)
        r2 = (d * d).sum(2)
        off = (r2 > 0) & (r2 < L * L / 4)
        r = torch.where(off, r2, torch.ones_like(r2)).sqrt()
        e = torch.erfc(alpha * r) / r
        g = (e + 2 * alpha / math.sqrt(math.pi) * torch.exp(-(alpha * r) ** 2)) / (r * r)
        qo = torch.where(off, q.expand_as(r), torch.zeros_like(r))
        phi[a:a + step] = (e * qo).sum(1)
        grad[a:a + step] = -torch.einsum("ij,ijk->ik", g * qo, d)
    k = torch.arange(-ksize, ksize + 1, device=x.device, dtype=torch.float64)
    k = torch.stack(torch.meshgrid(k, k, k, indexing="ij"), 3).reshape(-1, 3)
    k = k[(k * k).sum(1) > 0]
    kk = (k * k).sum(1)
    c = torch.exp(-(math.pi / (alpha * L)) ** 2 * kk) / (math.pi * L * kk)
    step = max(1, (1 << 26) // n)
    for a in range(0, len(k), step):
        th = (2 * math.pi / L) * (x @ k[a:a + step].T)
        co, si = torch.cos(th), torch.sin(th)
        re, im = q @ co, q @ si
        phi += co @ (c[a:a + step] * re) + si @ (c[a:a + step] * im)
        w = (co * im - si * re) * c[a:a + step]
        grad += w @ ((2 * math.pi / L) * k[a:a + step])
    phi -= 2 * alpha / math.sqrt(math.pi) * q
    y = x - L / 2
    mu = q @ y
    s = 4 * math.pi / (3 * L ** 3)
    phi += s * (y @ mu) - 0.5 * s * (q @ (y * y).sum(1))
    grad += s * mu
    return phi, grad


def exact(case, seed):
    """Potential and gradient by direct or Ewald sums, up to 2^18 bodies; for
    the adjoint in free space also dL/dq and dL/dx."""
    n, L = case["n"], case["cycle"]
    if n > 1 << 18:
        return None
    x, q, w = _bodies(case, seed)
    if case["images"] == 0:
        phi, grad = _direct(x, q)
    else:
        phi, grad = _ewald(x, q, L)
    scale = 1 / (4 * math.pi)
    out = []
    if case["call"] == "adjoint":
        out = [None, None]
        if case["images"] == 0:
            psi, dpsi = _direct(x, w)
            out = [psi * scale, (w[:, None] * grad + q[:, None] * dpsi) * scale]
    if case["dipole"]:
        y = x - L / 2
        mu = q @ y
        s = 4 * math.pi / (3 * L ** 3)
        phi = phi - (s * (mu @ mu) / n / q if case["dipole"] == 1 else s * (y @ mu))
        grad = grad - s * mu
    out = [phi * scale, grad * scale] + out
    if case["call"] in ("solve", "evaluate"):
        out = [None if v is None else v.cpu().numpy() for v in out]
    return out
