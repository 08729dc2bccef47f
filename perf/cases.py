"""The workloads the framework's speed is followed on.

Each case is one call, or one flow step, of the public interface at the sizes
the framework is used at, with the repository's own seeded mechanisms (9
species / 21 reactions and 53 species / 325 reactions) and cell distributions:

  reactor   integrate_host: the constant-pressure reactor of a few cells on
            host buffers (the 0-D application and the per-cell solve)
  flow      ChemistrySource.solveUpdate: one flow step of a block of cells,
            the call a flow solver spends its chemistry time in
  source    Mechanism.source_terms: explicit source terms of every cell
  implicit  Mechanism.source_terms_imp: point-implicit source terms
  jacobian  Mechanism.rhs_jacobian: f and J for a host-side implicit solver
  props     Mechanism.properties: thermodynamic and transport properties
  predict   Surrogate.features + predict: the learned step's inference
  grad      MLP.grad: loss and gradients of one training batch
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from openhurricane_b200 import synth, workloads
from openhurricane_b200.chemistry import ChemistrySource, Flow, Mechanism, integrate_host
from openhurricane_b200.surrogate import MLP, Surrogate

# Newton iterations a cell takes per flow step at the solver's options (means
# measured with the integrator's own counters), for the work of the flow cases
NEWTON = {"batched": 4800.0, "small": 1950.0, "large": 3500.0}

# A few cells in a thousand take 10 to 100 times the mean number of Newton
# iterations (up to 700,000 of them); the flow solver bounds the work of a
# cell and step with max_newton_total and gets such cells flagged.
CAP = {"batched": 40000, "small": 20000, "large": 6000}


def listed():
    return [
        # the per-cell solve: one 0-D reactor, latency of the whole call
        {"name": "reactor_9sp_1", "kind": "reactor", "cells": "small", "n": 1, "dt": 1e-6, "reactor": 0},
        # the smallest workload's block: Dirichlet states, a flow step of 1e-7 s
        {"name": "flow_9sp_4096", "kind": "flow", "cells": "small", "n": 4096, "dt": 1e-7, "reactor": 0},
        # ignition and near-equilibrium cells mixed: a block of the 1M-cell workload at its 1e-5 s
        {"name": "flow_9sp_batched", "kind": "flow", "cells": "batched", "n": 12288, "dt": 1e-5, "reactor": 0},
        # a block of the large mechanism
        {"name": "flow_53sp", "kind": "flow", "cells": "large", "n": 768, "dt": 1e-7, "reactor": 0},
        # the constant-volume reactor option on a ragged block
        {"name": "flow_9sp_volume", "kind": "flow", "cells": "small", "n": 1001, "dt": 1e-7, "reactor": 1},
        # explicit source terms: a whole domain, a domain of the large mechanism, a small ragged block
        {"name": "source_9sp_1m", "kind": "source", "cells": "batched", "n": 1048576},
        {"name": "source_53sp", "kind": "source", "cells": "large", "n": 65536},
        {"name": "source_9sp_257", "kind": "source", "cells": "small", "n": 257},
        # point-implicit source terms of a mid-size domain
        {"name": "implicit_9sp", "kind": "implicit", "cells": "batched", "n": 262144},
        # Jacobians of a ragged batch for a host-side implicit solver
        {"name": "jacobian_53sp", "kind": "jacobian", "cells": "large", "n": 8191},
        # thermodynamic and transport properties of a domain
        {"name": "props_53sp", "kind": "props", "cells": "large", "n": 65536},
        # the learned step's inference on a block
        {"name": "predict_9sp", "kind": "predict", "cells": "batched", "n": 131072},
    ]


def _log_size(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n | 1 if rng.random() < 0.7 else n))


def draw(rng):
    kind = rng.choice(["reactor", "flow", "flow", "flow", "source", "source", "implicit", "jacobian",
                       "props", "predict", "grad"])
    if kind == "reactor":
        return {"kind": kind, "cells": rng.choice(["small", "large"]), "n": rng.randint(1, 16),
                "dt": rng.choice([1e-8, 1e-7, 1e-6]), "reactor": rng.randint(0, 1)}
    if kind == "flow":
        cells = rng.choice(["small", "batched", "large"])
        hi = {"small": 4096, "batched": 12288, "large": 768}[cells]
        return {"kind": kind, "cells": cells, "n": _log_size(rng, 32, hi),
                "dt": rng.choice([1e-6, 1e-5] if cells == "batched" else [1e-8, 1e-7]),
                "reactor": 1 if cells == "small" and rng.random() < 0.4 else 0}
    cells = rng.choice(["small", "batched", "large"])
    big = cells == "large"
    hi = {"source": 65536 if big else 1048576, "implicit": 16384 if big else 262144,
          "jacobian": 8192 if big else 131072, "props": 65536 if big else 1048576,
          "predict": 131072, "grad": 8192}[kind]
    if kind in ("predict", "grad") and big:
        cells = "small"
    return {"kind": kind, "cells": cells, "n": _log_size(rng, 64, hi)}


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _tables(which):
    return workloads.mechanism_files(which)[2]


def _mech_name(case):
    return "large" if case["cells"] == "large" else "small"


def _cells(case, seed):
    """T, p, rho, Y of the case's cells (numpy, seeded)."""
    n, which = case["n"], case["cells"]
    if which == "batched":
        w = workloads.make_batched(n, seed=7919 * seed + 5, pool=min(1024, max(8, n)))
        return w.T, w.p, w.rho, w.Y
    t = _tables(_mech_name(case))
    c = (workloads.large_cells if which == "large" else workloads.small_cells)(n, seed=7919 * seed + 5)
    return c.T, c.p, synth.mixture_density(t.W, c), c.Y


def _dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _opts(case):
    return dict(workloads.SOLVER_OPTS, reactor=case["reactor"], max_newton_total=CAP[case["cells"]])


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    t = _tables(_mech_name(case))
    if kind == "grad":
        # a training batch of normalised features and targets, and the network
        # with the surrogate's stated sizes
        g = torch.Generator(device="cuda").manual_seed(seed)
        net = MLP(t.nsp + 3, t.nsp + 1, 3, 256, max_batch=8192, seed=seed)
        X = torch.randn(n, t.nsp + 3, generator=g, device="cuda")
        A = torch.randn(t.nsp + 3, t.nsp + 1, generator=g, device="cuda") / math.sqrt(t.nsp + 3.0)
        return {"case": case, "net": net, "X": X, "Y": torch.tanh(X @ A).contiguous()}
    T, p, rho, Y = _cells(case, seed)
    mech = Mechanism(t)
    s = {"case": case, "mech": mech, "T0": T, "p0": p, "rho0": rho, "Y0": Y}
    dt = np.full(n, case.get("dt", 1e-5))
    if kind == "reactor":
        s["dt"] = dt
        return s
    s.update(T=_dev(T), p=_dev(p), rho=_dev(rho), Y=_dev(Y))
    if kind == "flow":
        s["init"] = [s["T"].clone(), s["rho"].clone(), s["Y"].clone()]
        s["dt"] = _dev(dt)
        s["flow"] = Flow(s["T"], s["p"], s["rho"], s["Y"])
        s["cs"] = ChemistrySource(mech, s["flow"], **_opts(case))
        s["cs"].dtInit = s["dt"].clone()
    elif kind == "jacobian":
        s["c"] = (s["rho"][None] * s["Y"] / _dev(t.W)[:, None]).contiguous()
    elif kind == "predict":
        sur = Surrogate(mech, max_batch=65536, seed=seed)
        s["dt"] = _dev(dt * np.exp(np.random.default_rng(seed).uniform(-1.0, 1.0, n)))
        # normalisation as after training: input statistics of the cells, and
        # increments of the size a flow step makes
        raw = sur.raw_features(s["T"], s["p"], s["Y"], s["dt"])
        sd = raw.std(0)
        sur.in_mean = raw.mean(0).contiguous()
        sur.in_istd = torch.where(sd > 1e-12, 1.0 / sd, torch.ones_like(sd)).contiguous()
        sur.out_std = torch.full_like(sur.out_std, 1e-3)
        sur.out_std[0] = 10.0
        s["sur"] = sur
    return s


def run(s):
    case = s["case"]
    kind, mech = case["kind"], s.get("mech")
    if kind == "reactor":
        o = integrate_host(mech, s["T0"].copy(), s["p0"], s["rho0"].copy(), s["Y0"].copy(), s["dt"],
                           **_opts(case))
        return {k: o[k] for k in ("T", "rho", "Y", "status")}
    if kind == "flow":
        # the flow solver's fields at the start of the chemistry step
        for a, b in zip((s["T"], s["rho"], s["Y"]), s["init"]):
            a.copy_(b)
        s["cs"].dtInit.copy_(s["dt"])
        s["cs"].solveUpdate(s["dt"], 1.0)
        return {"T": s["T"], "rho": s["rho"], "Y": s["Y"], "status": s["cs"].status}
    if kind == "source":
        return mech.source_terms(s["T"], s["p"], s["rho"], s["Y"])
    if kind == "implicit":
        return mech.source_terms_imp(s["T"], s["p"], s["rho"], s["Y"])
    if kind == "jacobian":
        return mech.rhs_jacobian(s["c"], s["T"], s["p"])
    if kind == "props":
        return mech.properties(s["T"], s["p"], s["Y"])
    if kind == "predict":
        X = s["sur"].features(s["T"], s["p"], s["Y"], s["dt"])
        mean, spread = s["sur"].predict(X)
        return X, mean, spread
    loss, g = s["net"].grad(s["X"], s["Y"])
    return loss, g


# ------------------------------------------------------------------ work
@functools.lru_cache(maxsize=None)
def _flops(which):
    return workloads.flop_model(_tables(which))


def work(case):
    kind, n = case["kind"], case["n"]
    t = _tables(_mech_name(case))
    nsp, n1 = t.nsp, t.nsp + 1
    f = _flops(_mech_name(case))
    b = 8.0 * n
    if kind in ("reactor", "flow"):
        it = NEWTON[case["cells"]] * n
        # T, rho, Y in and out, p, dt in, the sub-step in and out, the status out
        return {"bytes": b * (2 * nsp + 8.5), "flops": it * (f["jac"] + f["lu"] + f["solve"])}
    if kind == "source":
        return {"bytes": b * (2 * nsp + 3), "flops": n * f["rhs"]}
    if kind == "implicit":
        return {"bytes": b * (3 * nsp + 2), "flops": n * f["jac"]}
    if kind == "jacobian":
        return {"bytes": b * (nsp + 2 + n1 + n1 * n1), "flops": n * f["jac"]}
    if kind == "props":
        # viscosity ratios, Wilke factors and diffusion pairs: about 20 operations a pair
        return {"bytes": b * (3 * nsp + 5), "flops": n * (20.0 * nsp * nsp + 100.0 * nsp)}
    w, n_in, n_out = 256, nsp + 3, nsp + 1
    mac = n_in * w + 2 * w * w + w * n_out
    if kind == "predict":
        return {"bytes": b * (nsp + 3) + 4.0 * n * (n_in + n_out + 1) + 3 * 4.0 * mac,
                "flops": 3 * 2.0 * mac * n}
    return {"bytes": 4.0 * n * (n_in + n_out) + 8.0 * mac, "flops": 6.0 * mac * n}


# Tolerances, about four times what was measured. The integrations: the
# library's kernel families against each other, and one family against itself
# from mass fractions one unit in the last place away, differ by up to 3.5e-5
# (9 species, one cell by 9e-3 of the root mean square) and 1.5e-3 (53
# species, one cell by 4.4e-2) at the solver's rtol of 1e-4; up to 0.6 % of
# the cells' status words change where a cell stops near its iteration bound.
# Source terms and Jacobians lie within 1e-12 of `exact` (sums that cancel
# near equilibrium), the 16-bit network within 3.3e-3.
def tolerance(case):
    kind = case["kind"]
    if kind in ("reactor", "flow"):
        big = case["cells"] == "large"
        return {"rel": 6e-3 if big else 1e-3, "max": 0.2, "differ": 0.01}
    if kind == "predict":
        return {"rel": 1e-2, "max": 0.3}
    if kind == "grad":
        return {"rel": 2e-2, "max": 0.6}
    return {"rel": 5e-12, "max": 1e-9}


# ------------------------------------------------------------------ exact
def _thermo(t, T):
    """Molar cp, h, dcp/dT, G0, dG0/dT and the mass-basis cp, h of every species, [nsp, n]."""
    W = _dev(t.W)[:, None]
    hi = T[None] >= _dev(t.Trange[:, 1])[:, None]
    a = [torch.where(hi, _dev(t.nasa[:, 1, k])[:, None], _dev(t.nasa[:, 0, k])[:, None]) for k in range(7)]
    T = T[None]
    lT = torch.log(T)
    cp = a[0] + T * (a[1] + T * (a[2] + T * (a[3] + T * a[4])))
    h = T * (a[0] + T * (a[1] / 2 + T * (a[2] / 3 + T * (a[3] / 4 + T * a[4] / 5)))) + a[5]
    s = a[0] * lT + T * (a[1] + T * (a[2] / 2 + T * (a[3] / 3 + T * a[4] / 4))) + a[6]
    dcp = a[1] + T * (2 * a[2] + T * (3 * a[3] + T * 4 * a[4]))
    return cp * W, h * W, dcp * W, (h - T * s) * W, -s * W, cp, h


_RU = 1.380649e-23 * 6.02214076e23 * 1e3
_PATM = 101325.0


def _kinetics(t, c, T, jac):
    """omega [nsp, n] and, with jac, d omega/d(c, T) [nsp, nsp + 1, n], for the
    Arrhenius, third-body, Lindemann and Troe reactions of the two mechanisms."""
    nsp, n = c.shape
    cp, h, dcp, G, dG = _thermo(t, T)[:5]
    om = torch.zeros_like(c)
    J = torch.zeros((nsp, nsp + 1, n), dtype=c.dtype, device=c.device) if jac else None
    lT, ln10 = torch.log(T), math.log(10.0)
    for r in range(t.nrc):
        kind = int(t.rate_type[r])
        A, b, Ta = (float(v) for v in t.arr[r])
        k = A * torch.exp(b * lT - Ta / T)
        dk = k * (b + Ta / T) / T
        eff = _dev(t.eff[r])
        M = (eff[:, None] * c).sum(0) if kind else None
        dkM = None
        if kind == 1:
            dkM, k, dk = k, k * M, dk * M
        elif kind >= 2:
            A0, b0, Ta0 = (float(v) for v in t.arr0[r])
            k0 = A0 * torch.exp(b0 * lT - Ta0 / T)
            Pr = k0 * M / k
            dlPr = (b0 + Ta0 / T) / T - (b + Ta / T) / T       # d ln Pr / dT
            F, dlF_P, dlF_T = torch.ones_like(T), torch.zeros_like(T), torch.zeros_like(T)
            if kind >= 3:
                al, T3, T1, T2 = (float(v) for v in t.troe[r])
                e1, e2 = (1 - al) * torch.exp(-T / T3), al * torch.exp(-T / T1)
                e3 = torch.exp(-T2 / T) if kind == 4 else torch.zeros_like(T)
                Fc = e1 + e2 + e3
                lf, dlf = torch.log10(Fc), (-e1 / T3 - e2 / T1 + e3 * T2 / T ** 2) / (Fc * ln10)
                u = torch.log10(Pr) - 0.4 - 0.67 * lf
                v = 0.75 - 1.27 * lf - 0.14 * u
                x = u / v
                F = 10.0 ** (lf / (1 + x * x))
                g = -lf * 2 * x / (1 + x * x) ** 2            # d log10 F / dx
                xu, xl = (v + 0.14 * u) / v ** 2, 1.27 * u / v ** 2
                dlF_P = g * xu                                 # d ln F / d ln Pr
                dlF_T = ln10 * (dlf / (1 + x * x) + g * (xu * -0.67 + xl) * dlf)
            w = Pr / (1 + Pr) * F
            dkM = k * w * (1 / (1 + Pr) + dlF_P) / M
            dk = dk * w + k * w * ((1 / (1 + Pr) + dlF_P) * dlPr + dlF_T)
            k = k * w
        fi, bi = [int(i) for i in t.fidx[r, :t.nf[r]]], [int(i) for i in t.bidx[r, :t.nb[r]]]
        nuf, nub = [float(v) for v in t.fnu[r]], [float(v) for v in t.bnu[r]]
        of, ob = [float(v) for v in t.ford[r]], [float(v) for v in t.bord[r]]
        side = []
        for idx, order in ((fi, of), (bi, ob)):
            prod = torch.ones_like(T)
            for i, o in zip(idx, order):
                prod = prod * c[i] ** o
            part = []
            for a, (i, o) in enumerate(zip(idx, order)):
                d = o * c[i] ** (o - 1) if o != 1.0 else torch.ones_like(T)
                for e, (j, q) in enumerate(zip(idx, order)):
                    d = d * c[j] ** q if e != a else d
                part.append((i, d))
            side.append((prod, part))
        dGr = sum(v * G[i] for i, v in zip(bi, nub)) - sum(v * G[i] for i, v in zip(fi, nuf))
        dHr = sum(v * h[i] for i, v in zip(bi, nub)) - sum(v * h[i] for i, v in zip(fi, nuf))
        S = sum(nub[:len(bi)]) - sum(nuf[:len(fi)])
        iK = torch.exp(dGr / (_RU * T)) * (_RU * T / _PATM) ** S if int(t.reversible[r]) else torch.zeros_like(T)
        q = k * side[0][0] - k * iK * side[1][0]
        nu = torch.zeros(nsp, dtype=c.dtype, device=c.device)
        for i, v in zip(fi, nuf):
            nu[i] -= v
        for i, v in zip(bi, nub):
            nu[i] += v
        rows = torch.nonzero(nu).flatten().tolist()
        for i in rows:
            om[i] += nu[i] * q
        if not jac:
            continue
        # the reference's d ln Kp / dT has the opposite sign, and the interface keeps it
        diK = iK * (S / T + dHr / (_RU * T ** 2))
        dq = {nsp: dk * (side[0][0] - iK * side[1][0]) - k * diK * side[1][0]}
        for i, d in side[0][1]:
            dq[i] = dq.get(i, 0) + k * d
        for i, d in side[1][1]:
            dq[i] = dq.get(i, 0) - k * iK * d
        net = side[0][0] - iK * side[1][0]
        for i in rows:
            for j, d in dq.items():
                J[i, j] += nu[i] * d
            if dkM is not None:
                J[i, :nsp] += nu[i] * eff[:, None] * (dkM * net)[None]
    return om, J


def _exact_jacobian(t, c, T):
    om, J = _kinetics(t, c, T, True)
    cp, h, dcp = _thermo(t, T)[:3]
    C, dC = (c * cp).sum(0), (c * dcp).sum(0)
    dT = -(om * h).sum(0) / C
    row = -((J * h[:, None]).sum(0))                            # [nsp + 1, n]
    row[:-1] -= cp * dT[None]
    row[-1] -= (om * cp).sum(0) + dC * dT
    full = torch.cat([J, (row / C)[None]], 0)
    return torch.cat([om, dT[None]], 0).T.contiguous(), full.permute(2, 0, 1).contiguous()


def _exact_props(t, T, p, Y):
    W, (cpm, hm) = _dev(t.W)[:, None], _thermo(t, T)[5:]
    X = Y / W
    X = X / X.sum(0)
    eps, sg = _dev(t.eps_k), _dev(t.sigma)
    Ts = T[None] / eps[:, None]
    mu = 2.6693e-6 * torch.sqrt(W * T) / (sg[:, None] ** 2 * (1.147 * Ts ** -0.145 + (Ts + 0.5) ** -2))
    kap = mu * (cpm + 1.25 * _RU / W)
    num, numk, D = torch.zeros_like(T), torch.zeros_like(T), torch.empty_like(Y)
    for i in range(t.nsp):
        wr = W[i] / W
        phi = (1 + torch.sqrt(mu[i] / mu) * wr ** -0.25) ** 2 / torch.sqrt(8 * (1 + wr))
        den = (X * phi).sum(0)
        num += X[i] * mu[i] / den
        numk += X[i] * kap[i] / den
        Ts = T[None] / torch.sqrt(eps[i] * eps)[:, None]
        om = Ts ** -0.145 + (Ts + 0.5) ** -2          # the reference's diffusion form has no prefactor
        s2 = (0.5 * (sg[i] + sg))[:, None] ** 2
        Dij = 1.858e-7 * T ** 1.5 * torch.sqrt(1 / W[i] + 1 / W) / (s2 * om) * _PATM / p
        q = X / Dij
        D[i] = (1 - X[i]) / (q.sum(0) - q[i])
    return {"ha": hm, "cp": (Y * cpm).sum(0), "mu": num, "kappa": numk, "D": D}


def _layers(net):
    theta, off, out = torch.tensor(net.get_params(), device="cuda").double(), 0, []
    for o, i in net.shapes():
        out.append((theta[off:off + o * i].view(o, i), theta[off + o * i:off + o * i + o]))
        off += o * i + o
    return out


def _net64(layers, X):
    for k, (W, b) in enumerate(layers):
        X = torch.nn.functional.linear(X, W, b)
        X = torch.nn.functional.gelu(X) if k + 1 < len(layers) else X
    return X


def exact(case, seed):
    kind = case["kind"]
    if kind in ("reactor", "flow"):
        # thousands of dependent Newton iterations a cell with the solver's
        # adaptive steps: minutes in plain torch
        return None
    s, t = prepare(case, seed), _tables(_mech_name(case))
    if kind == "grad":
        layers = [(W.requires_grad_(), b.requires_grad_()) for W, b in
                  [(W.detach().clone(), b.detach().clone()) for W, b in _layers(s["net"])]]
        loss = ((_net64(layers, s["X"].double()) - s["Y"].double()) ** 2).mean()
        loss.backward()
        return float(loss), torch.cat([torch.cat([W.grad.flatten(), b.grad]) for W, b in layers]).cpu().numpy()
    T, p, rho, Y = s["T"], s["p"], s["rho"], s["Y"]
    W = _dev(t.W)[:, None]
    if kind == "source":
        return _kinetics(t, rho[None] * Y / W, T, False)[0] * W
    if kind == "implicit":
        out = []
        for k in range(0, T.shape[0], 65536):
            q = slice(k, k + 65536)
            Tk, Yk, rk = T[q], Y[:, q], rho[q]
            om, J = _kinetics(t, rk[None] * Yk / W, Tk, True)
            cpm, hm = _thermo(t, Tk)[5:]
            e = hm - _RU / W * Tk
            cv = (Yk * (cpm - _RU / W)).sum(0)
            L = t.nsp - 1
            d = torch.stack([J[i, i] - W[i] / W[L] * J[i, L] + J[i, -1] * W[i] * (e[L] - e[i]) / (rk * cv)
                             for i in range(L)])
            out.append((om * W, d))
        return torch.cat([a for a, _ in out], 1), torch.cat([b for _, b in out], 1)
    if kind == "jacobian":
        parts = [_exact_jacobian(t, s["c"][:, k:k + 4096], T[k:k + 4096]) for k in range(0, T.shape[0], 4096)]
        return torch.cat([a for a, _ in parts]), torch.cat([b for _, b in parts])
    if kind == "props":
        return _exact_props(t, T, p, Y)
    sur = s["sur"]
    X = (sur.raw_features(T, p, Y, s["dt"]) - sur.in_mean) * sur.in_istd
    preds = torch.stack([_net64(_layers(m), X) for m in sur.nets])
    rng = (preds.amax(0) - preds.amin(0)) * sur.out_std
    return X, preds.mean(0), torch.maximum(rng[:, 0] / sur.spread_T, rng[:, 1:].amax(1) / sur.spread_Y)
