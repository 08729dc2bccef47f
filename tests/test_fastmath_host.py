"""The kernels' exponential, logarithm and fall-off forms
(openhurricane_b200/csrc/fastmath.cuh) compiled for the host: the functions
against exact values, within one unit in the last place, and at the limits of their
range; the fall-off
forms against the reference's formulas (fallOffFunctions.cpp:81-157,
unimolecularFallOffRR.cpp:37-91) as written there."""
import math
import os
import shutil
import subprocess
from decimal import Decimal, localcontext

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
TINY = 1e-15


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("fastmath") / "fastmath")
    inc = os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"
    subprocess.check_call([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", inc, "-o", out,
                           os.path.join(HERE, "cpp", "fastmath.cpp")])
    return out


def _run(exe, kind, xs):
    txt = "\n".join(f"{kind} {float(x)!r}" for x in xs) + "\n"
    r = subprocess.run([exe], input=txt, capture_output=True, text=True, check=True)
    return np.array([float(v) for v in r.stdout.split()])


def _within_one_ulp(xs, got, exact):
    with localcontext() as ctx:
        ctx.prec = 50
        for x, g in zip(xs, got):
            ref = exact(Decimal(float(x)))
            assert abs(Decimal(float(g)) - ref) <= Decimal(math.ulp(float(ref))), (x, g)


def test_exp_within_one_ulp(exe):
    rng = np.random.default_rng(0)
    half = math.log(2.0) / 2
    xs = np.concatenate([rng.uniform(-1, 1, 2000), rng.uniform(-60, 60, 2000), rng.uniform(-699.9, 699.9, 2000),
                         half * (2 * rng.integers(-900, 900, 500) + 1) * (1 + rng.uniform(-1e-12, 1e-12, 500)),
                         [0.0, -0.0, 1e-300, -1e-300, 1e-17, half, -half, 699.999, -699.999]])
    got = _run(exe, "E", xs)
    _within_one_ulp(xs, got, lambda d: d.exp())
    assert np.array_equal(_run(exe, "X", xs), got)


def test_log_within_one_ulp(exe):
    rng = np.random.default_rng(1)
    s = math.sqrt(0.5)
    xs = np.concatenate([rng.uniform(200, 6000, 2000), 10.0 ** rng.uniform(-300, 300, 2000),
                         1.0 + rng.uniform(-1e-3, 1e-3, 2000), 2.0 ** rng.integers(-1000, 1000, 200),
                         s * 2.0 ** rng.integers(-20, 20, 500) * (1 + rng.uniform(-1e-9, 1e-9, 500)),
                         [1.0, 1 + 2.0 ** -52, 1 - 2.0 ** -53, 2.2250738585072014e-308, 1.7976931348623157e308]])
    _within_one_ulp(xs, _run(exe, "L", xs), lambda d: d.ln())


def test_limits_infinities_and_nan(exe):
    xs = [710.0, 800.0, 1e308, math.inf, -746.0, -801.0, -1e308, -math.inf]
    for kind in "EX":
        assert np.array_equal(_run(exe, kind, xs), np.array([math.inf] * 4 + [0.0] * 4))
    # below the normal range the result rounds twice: one unit of the smallest number
    low = np.linspace(-745.0, -708.0, 200)
    assert (np.abs(_run(exe, "E", low) - np.exp(low)) <= 5e-324 + 2.3e-16 * np.exp(low)).all()
    _within_one_ulp([700.0, 709.0, 709.78], _run(exe, "E", [700.0, 709.0, 709.78]), lambda d: d.exp())
    assert np.array_equal(_run(exe, "L", [0.0, -0.0, math.inf]), np.array([-math.inf, -math.inf, math.inf]))
    _within_one_ulp([5e-324, 1e-310], _run(exe, "L", [5e-324, 1e-310]), lambda d: d.ln())
    assert np.isnan(_run(exe, "E", [math.nan])).all() and np.isnan(_run(exe, "X", [math.nan])).all()
    assert np.isnan(_run(exe, "L", [math.nan, -1.0])).all()


def _reference(troe, al, T3, T1, T2, four, T, ratio, M, dlr):
    """k0 M / kinf etc. as the reference writes them, with kinf = 1."""
    Pr = ratio * M
    F, fabc, dFdT = 1.0, 0.0, 0.0
    dPrdT = Pr * dlr
    if troe:
        e1, e2, e3 = math.exp(-T / T3), math.exp(-T / T1), math.exp(-T2 / T) if four else 0.0
        Fc = max((1 - al) * e1 + al * e2 + e3, TINY)
        dFc = (1 - al) * e1 / -T3 + al * e2 / -T1 + (e3 * T2 / T ** 2 if four else 0.0)
        lf = math.log10(Fc)
        lp = math.log10(max(Pr, TINY))
        c, n, d = -0.4 - 0.67 * lf, 0.75 - 1.27 * lf, 0.14
        x = (lp + c) / (n - d * (lp + c))
        F = 10.0 ** (lf / (1 + x * x))
        nm = n - d * (lp + c)
        inv = (lp + c) / nm
        s1 = 1 + inv * inv
        fabc = F * (-lf / s1 ** 2) * (2 * (lp + c) / nm ** 2) * (1 + d * inv)
        dlf = dFc / (Fc * math.log(10.0))
        Dc, Dn = -0.67 * dlf, -1.27 * dlf
        dlp = dPrdT / Pr / math.log(10.0)
        dPP = 2 * (lp + c) / nm ** 2 * ((dlp + Dc) - inv * (Dn - d * (dlp + Dc)))
        dFdT = F * math.log(10.0) * (dlf / s1 - lf / s1 ** 2 * dPP)
    w = Pr / (1 + Pr) * F
    g = ratio * (1 / (Pr * (1 + Pr)) + fabc / Pr / F)
    dT = dPrdT / (Pr * (1 + Pr)) + dFdT / F
    return w, (g if M > TINY else 0.0), (dT if M > TINY else 0.0)


def test_fall_off_matches_the_reference_formulas(exe):
    rng = np.random.default_rng(5)
    rows = []
    for k in range(600):
        M = 10.0 ** rng.uniform(-16, 1)
        rows.append((float(k % 3 > 0), rng.uniform(0.05, 0.95), 10 ** rng.uniform(1, 4), 10 ** rng.uniform(1, 4),
                     10 ** rng.uniform(2, 4), float(k % 3 > 1), rng.uniform(250, 4000), 10.0 ** rng.uniform(-8, 8) / M,
                     M, rng.uniform(-0.05, 0.05)))
    txt = "\n".join("F " + " ".join(repr(float(v)) for v in r) for r in rows) + "\n"
    out = subprocess.run([exe], input=txt, capture_output=True, text=True, check=True).stdout
    got = np.array([[float(x) for x in l.split()] for l in out.strip().splitlines()])
    for r, g in zip(rows, got):
        ref = _reference(r[0] != 0, *r[1:5], r[5] != 0, *r[6:])
        # the exponent of F (up to 35) and the differences of the derivatives' terms
        # lose two to three digits of 16 in either form
        scale = (abs(ref[0]), abs(ref[1]), abs(r[9]) + abs(ref[2]) + 1e-3)
        for a, b, s in zip(g, ref, scale):
            assert abs(a - b) <= 1e-12 * s + 1e-300, (r, g, ref)
