"""The work that users of this library have it do, as cases that can be timed.

A case is a dict of plain values:

  mode      what one pass is:
            "step"     a new FMM on a new point set: FMM(x, y, ...), build_tree, precompute,
                       build_expansions(tau), evaluate_to_points(x, y, True), as the
                       reference's examples run it;
            "rebuild"  the same four calls on an FMM object that the program keeps (a loop
                       that moves its points in place);
            "apply"    a new density on a tree and operators that are there already
                       (an iterative solver): build_expansions(tau), evaluate_to_points;
            "replay"   the same apply captured as a CUDA graph (the serving loop);
            "targets"  evaluate_to_points at m other points (a field on a grid or a plot)
                       from expansions that are there already
  kernel    "laplace", "k0" (modified Helmholtz, wavenumber k) or "h0" (Helmholtz, complex)
  points    "uniform" in [-1, 1]^2, "mixture" (16 Gaussians and 20% of the points on the unit
            circle) or "annulus" (0.5 < r < 1), the clouds of the benchmark configurations
  n, m      source points; separate targets
  nequiv, ncutoff, precision, planned    options of FMM
  host      points, densities and results are numpy arrays in host memory
"""
import math

import numpy as np
import torch

import pykifmm2d_b200 as P

DEV = "cuda:0"


def _case(name, mode, kernel, points, n, nequiv, ncutoff, precision, k=0.0, m=0, planned=False, host=False):
    c = {"mode": mode, "kernel": kernel, "k": k, "points": points, "n": n, "m": m, "nequiv": nequiv,
         "ncutoff": ncutoff, "precision": precision, "planned": planned, "host": host}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest request of a serving stream, one density of an iterative solve on it: all
        # launches and latency
        _case("apply_1k_laplace_fp64", "apply", "laplace", "mixture", 1000, 32, 64, "fp64"),
        # a small problem from its points to its potentials, as the examples call it
        _case("step_20k_laplace_fp64", "step", "laplace", "uniform", 20_000, 24, 64, "fp64"),
        # one density of a medium-sized serving request, as the server replays it
        _case("replay_30k_laplace_mixed", "replay", "laplace", "mixture", 30_001, 32, 64, "mixed"),
        # a middle-sized problem called with numpy arrays on the host: copies and a new plan each time
        _case("host_step_200k_laplace_mixed", "step", "laplace", "mixture", 200_003, 32, 64, "mixed", host=True),
        # the headline workload: every part of the path on an adaptive tree
        _case("rebuild_1m_laplace_mixed", "rebuild", "laplace", "mixture", 1_000_000, 32, 64, "mixed"),
        # repeated densities in the default precision
        _case("apply_1m_laplace_fp64", "apply", "laplace", "mixture", 1_000_000, 32, 64, "fp64"),
        # the largest full step: four million points, a new plan
        _case("step_4m_laplace_mixed", "step", "laplace", "uniform", 4_000_000, 32, 64, "mixed"),
        # the screened kernel at its benchmark size, repeated densities
        _case("apply_2m_k0_mixed", "apply", "k0", "annulus", 2_000_000, 40, 48, "mixed", k=10.0),
        # the screened kernel in the default precision, from its points
        _case("rebuild_300k_k0_fp64", "rebuild", "k0", "annulus", 299_993, 40, 48, "fp64", k=10.0),
        # a field evaluated away from its sources
        _case("targets_3m_laplace_mixed", "targets", "laplace", "mixture", 300_000, 32, 64, "mixed", m=2_999_999),
        # complex densities and kernel (the Helmholtz example's options)
        _case("apply_150k_h0_complex", "apply", "h0", "uniform", 150_000, 24, 50, "fp64", k=2.0),
        # repeated densities with the kernel values kept as matrices
        _case("planned_500k_k0_fp64", "apply", "k0", "annulus", 500_001, 40, 48, "fp64", k=10.0, planned=True),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | (rng.random() < 0.5)

    kind = rng.choice(["laplace"] * 5 + ["k0"] * 3 + ["h0"])
    mode = rng.choice(["step", "rebuild", "apply", "replay", "targets"])
    points = rng.choice(["uniform", "mixture", "annulus"])
    precision, planned, host, k, m = rng.choice(["fp64", "mixed"]), False, False, 0.0, 0
    if kind == "laplace":
        nequiv, ncutoff = rng.choice([(24, 64), (32, 64), (32, 50), (48, 50)])
        top = 1_000_000 if precision == "fp64" else 3_000_000
    elif kind == "k0":
        nequiv, ncutoff, k = rng.choice([32, 40]), rng.choice([48, 64]), rng.choice([1.0, 10.0, 50.0])
        top = 300_000 if precision == "fp64" else 1_000_000
    else:
        nequiv, ncutoff, k, precision = rng.choice([24, 32]), 50, rng.choice([2.0, 10.0]), "fp64"
        top = 150_000
    if mode == "replay":
        top = 300_000 if kind != "h0" else 100_000
    if mode == "targets":
        top = {"laplace": 500_000, "k0": 100_000, "h0": 30_000}[kind]
        m = size(1000, {"laplace": 3_000_000, "k0": 300_000, "h0": 50_000}[kind])
    if mode == "apply" and kind != "h0":
        planned = rng.random() < 0.25
        top = min(top, 500_000) if planned else top
    if mode in ("step", "rebuild", "apply"):
        host = rng.random() < 0.2
    return _case(None, mode, kind, points, size(1000, top), nequiv, ncutoff, precision, k, m, planned, host)


# ------------------------------------------------------------------ inputs
def _cloud(kind, n, g):
    def u(lo, hi, size):
        return torch.rand(size, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo

    if kind == "uniform":
        return u(-1, 1, n), u(-1, 1, n)
    th = u(0, 2 * math.pi, n)
    if kind == "annulus":
        r = u(0.25, 1, n).sqrt()
        return r * th.cos(), r * th.sin()
    nc = n // 5
    cx, cy, sig = u(-1, 1, 16), u(-1, 1, 16), 10 ** u(-3, -1, 16)
    lab = torch.randint(0, 16, (n - nc,), generator=g, device=DEV)
    z = torch.randn((2, n - nc), generator=g, device=DEV, dtype=torch.float64)
    th = th[:nc]
    return (torch.cat([cx[lab] + sig[lab] * z[0], th.cos()]), torch.cat([cy[lab] + sig[lab] * z[1], th.sin()]))


def _inputs(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    n = case["n"]
    x, y = _cloud(case["points"], n, g)
    if case["kernel"] == "h0":
        t = torch.randn((n, 2), generator=g, device=DEV, dtype=torch.float64)
        tau = torch.view_as_complex(t).clone()
    else:
        tau = torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
    tx, ty = _cloud("uniform", case["m"], g) if case["m"] else (None, None)
    return x, y, tau, tx, ty


def _fmm(case, x, y, stream=None):
    kern = {"laplace": P.LaplaceKernel, "k0": lambda: P.ModifiedHelmholtzKernel(case["k"]),
            "h0": lambda: P.HelmholtzKernel(case["k"])}[case["kernel"]]()
    return P.FMM(x, y, P.Get_Kernel_Functions(kern), P.prepare_numba_functions_on_the_fly(kern), case["nequiv"],
                 case["ncutoff"], case["kernel"] == "h0", precision=case["precision"], planned=case["planned"],
                 stream=stream)


def prepare(case, seed):
    x, y, tau, tx, ty = _inputs(case, seed)
    if case["host"]:
        x, y, tau = (v.cpu().numpy() for v in (x, y, tau))
    s = {"case": case, "x": x, "y": y, "tau": tau, "tx": tx, "ty": ty}
    mode = case["mode"]
    if mode == "step":
        return s
    if mode == "replay":
        s["stream"] = torch.cuda.Stream(DEV)
        s["pot"] = torch.empty_like(tau)
        torch.cuda.synchronize()
        s["fmm"] = f = _fmm(case, x, y, s["stream"].cuda_stream)
        f.capture_apply(tau, s["pot"], True)
        return s
    s["fmm"] = f = _fmm(case, x, y)
    if mode in ("apply", "targets"):
        f.build_tree()
        f.precompute()
    if mode == "targets" or case["planned"]:
        # the targets' expansions; a planned apply lays its matrices out at the first density
        f.build_expansions(tau)
        if case["planned"]:
            f.evaluate_to_points(x, y, True)
    return s


def run(state):
    mode, x, y, tau = state["case"]["mode"], state["x"], state["y"], state["tau"]
    if mode == "replay":
        state["fmm"].replay()
        return state["pot"]
    if mode == "targets":
        return state["fmm"].evaluate_to_points(state["tx"], state["ty"], False)
    f = _fmm(state["case"], x, y) if mode == "step" else state["fmm"]
    if mode != "apply":
        f.build_tree()
        f.precompute()
    f.build_expansions(tau)
    return f.evaluate_to_points(x, y, True)


# -------------------------------------------------------------------- work
def work(case):
    n, m, q, cut = case["n"], case["m"], case["nequiv"], case["ncutoff"]
    val = 16 if case["kernel"] == "h0" else 8
    # a real kernel value and its product with a density: Laplace 8 flops, K0 and H0 about 40;
    # about 0.45 Ncutoff points in a leaf, 10 leaves' sources to a target, 27 boxes to a translation
    pair = 8 if case["kernel"] == "laplace" else 40
    per_leaf = 0.45 * cut
    leaves = n / per_leaf
    near = (10 if n > cut else 1) * min(per_leaf, n)
    if case["mode"] == "targets":
        return {"bytes": 24 * m + 24 * n + 8 * q * leaves, "flops": m * (q + near) * pair}
    flops = n * (2 * q + near) * pair + leaves * 1.33 * (27 + 2) * 2 * q * q * (4 if val == 16 else 1)
    size = 2 * val * n + (16 * n if case["mode"] in ("step", "rebuild") else 0)
    if case["planned"]:
        size += n * (2 * q + near) * 8
        flops = n * (2 * q + near) * 2
    return {"bytes": size, "flops": flops}


# ------------------------------------------------------------------- exact
def _pairs_limit(case):
    # about 20 seconds of direct sums
    return 1.1e12 if case["kernel"] == "laplace" else 1.0e11


def exact(case, seed):
    """The direct sum in 64 bits (pairs at distance 0 left out)."""
    x, y, tau, tx, ty = _inputs(case, seed)
    if tx is None:
        tx, ty = x, y
    if float(x.numel()) * tx.numel() > _pairs_limit(case):
        return None
    out = torch.empty(tx.numel(), dtype=tau.dtype, device=DEV)
    rows = max(1, min(tx.numel(), (1 << 23) // min(x.numel(), 8192)))
    for a in range(0, tx.numel(), rows):
        px, py = tx[a:a + rows, None], ty[a:a + rows, None]
        acc = torch.zeros(px.shape[0], dtype=tau.dtype, device=DEV)
        for b in range(0, x.numel(), 8192):
            d = px - x[None, b:b + 8192]
            r2 = d.mul_(d)
            e = py - y[None, b:b + 8192]
            r2.addcmul_(e, e)
            zero = r2 == 0
            t = tau[b:b + 8192]
            if case["kernel"] == "laplace":
                acc += (r2.masked_fill_(zero, 1.0).log_() @ t) * (-0.25 / math.pi)
            elif case["kernel"] == "k0":
                v = torch.special.modified_bessel_k0(r2.sqrt_().mul_(case["k"]))
                acc += (v.masked_fill_(zero, 0.0) @ t) / (2 * math.pi)
            else:
                z = r2.sqrt_().mul_(case["k"])
                re = torch.special.bessel_y0(z).mul_(-0.25).masked_fill_(zero, 0.0)
                im = torch.special.bessel_j0(z).mul_(0.25).masked_fill_(zero, 0.0)
                acc += torch.complex(re @ t.real - im @ t.imag, re @ t.imag + im @ t.real)
        out[a:a + rows] = acc
    return np.asarray(out.cpu()) if case["host"] else out
