"""Source terms, point-implicit terms, Jacobians and properties on the GPU
against the CPU oracle at the sizes where the lanes-per-cell and
block-per-cell kernels change shape: one cell, the edges of a block's cells,
each lane count's range, mechanisms on both sides of a column-block or row
limit, temperatures outside the fitted range, species that are absent.

Tolerance: sums of up to n_rxn products in another order, each term good to a
few units in the last place after an exponential of an argument of up to 200
(relative error 200 * 2^-53): 1e-11 of the largest magnitude in the row, and
1e-12 for the properties, whose terms are all positive."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# species, reactions, third-body, Troe: both sides of the integrators' and row
# blocks' limits (nsp + 1 = 16 | 17, 32 | 33, 55 | 56, 64)
MECHS = [(15, 45, 8, 3), (16, 50, 10, 4), (31, 120, 20, 6), (32, 120, 20, 6), (54, 300, 50, 12),
         (55, 300, 50, 12), (63, 400, 60, 20)]


def _dev():
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch.device("cuda:0")


def _tables(nsp, nrc, ntb, nt, tmp):
    from openhurricane_b200 import synth
    from openhurricane_b200.mechanism import compile_mechanism
    m = synth.make_mechanism(nsp, nrc, ntb, nt, seed=5 + nsp)
    return compile_mechanism(*synth.write_chemkin(m, str(tmp / f"m{nsp}")))


def _states(t, n, cold=False):
    from openhurricane_b200 import synth
    c = synth.dirichlet_cells(t.nsp, n, seed=n + t.nsp, T_range=(200.0, 5500.0) if cold else (800.0, 2800.0),
                              alpha=0.3)
    if cold:
        c.Y[:, ::3] = 0.0
        c.Y[0, ::3] = 0.25            # only two species present
        c.Y[t.nsp - 1, ::3] = 0.75
    return c, synth.mixture_density(t.W, c)


def _close(g, r, tol, axis, what):
    g = g.cpu().numpy()
    scale = np.abs(r).max(axis=axis, keepdims=True) + 1e-300
    assert (np.abs(g - r) / scale).max() <= tol, what


def _check(t, n, cold=False):
    from openhurricane_b200.chemistry import Mechanism
    from oracle import port, props_oracle, srcimp_oracle
    dev = _dev()
    c, rho = _states(t, n, cold)
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
    T, p, rh, Y = d(c.T), d(c.p), d(rho), d(c.Y)
    m = Mechanism(t)
    conc = rho[None] * c.Y / t.W[:, None]
    f, J = port.rhs_jac(port.MechDesc(t), conc, c.T, c.p)
    ref = srcimp_oracle.srcimp(t, c.T, c.p, rho, c.Y)
    _close(m.source_terms(T, p, rh, Y), ref["Ri"], 1e-11, 0, "source")
    Ri, diag = m.source_terms_imp(T, p, rh, Y)
    _close(Ri, ref["Ri"], 1e-11, 0, "implicit Ri")
    _close(diag, ref["diag"], 1e-11, 0, "diag")
    gf, gJ = m.rhs_jacobian(d(conc), T, p)
    _close(gf[:, :t.nsp], f[:, :t.nsp], 1e-11, 1, "f")
    # the temperature row is -sum_i h_i (row i) / C: its terms cancel, so their size sets the bar
    pr = props_oracle.properties(t, c.T, c.p, c.Y)
    hC = (np.abs(pr["ha"]) * t.W[:, None] / (rho * pr["cp"])).T            # [n, nsp]
    size = (np.abs(f[:, :t.nsp]) * hC).sum(axis=1)
    assert (np.abs(gf[:, t.nsp].cpu().numpy() - f[:, t.nsp]) <= 1e-11 * size).all()
    _close(gJ[:, :t.nsp], J[:, :t.nsp], 1e-11, 2, "J")
    size = (np.abs(J[:, :t.nsp]) * hC[:, :, None]).sum(axis=1).max(axis=1) + np.abs(J[:, t.nsp]).max(axis=1)
    assert (np.abs(gJ[:, t.nsp].cpu().numpy() - J[:, t.nsp]).max(axis=1) <= 1e-11 * size).all()
    gf2, none = m.rhs_jacobian(d(conc), T, p, jac=False)
    assert none is None
    _close(gf2[:, :t.nsp], f[:, :t.nsp], 1e-11, 1, "f alone")
    g = m.properties(T, p, Y)
    for k in ("ha", "cp", "mu", "kappa", "D"):
        _close(g[k], pr[k], 1e-12, 0 if pr[k].ndim == 2 else None, k)
    m.close()


@pytest.mark.parametrize("n", [1, 31, 33, 129])
@pytest.mark.parametrize("shape", MECHS, ids=lambda s: f"{s[0]}sp")
def test_mechanism_sizes(shape, n, tmp_path):
    _check(_tables(*shape, tmp_path), n)


@pytest.mark.parametrize("name", ["small", "large"])
@pytest.mark.parametrize("n", [1, 127, 2500, 20001])
def test_cell_counts(name, n, request):
    if name == "large" and n > 5000:
        n = 4801
    _check(request.getfixturevalue(name)["tables"], n)


@pytest.mark.parametrize("name", ["small", "large"])
def test_cold_hot_and_absent_species(name, request):
    _check(request.getfixturevalue(name)["tables"], 200, cold=True)


@pytest.mark.parametrize("shape", [(17, 60, 10, 4), (31, 120, 20, 6), (40, 200, 40, 10), (55, 300, 50, 12),
                                   (63, 400, 60, 20)], ids=lambda s: f"{s[0]}sp")
@pytest.mark.parametrize("reactor", [0, 1])
def test_block_per_cell_integration_vs_oracle(shape, reactor, tmp_path):
    """Both reactors, each size's column and row blocks; cells whose answer one
    unit in the last place does not move must agree (parity_util)."""
    from parity_util import check
    from openhurricane_b200.chemistry import ChemistrySource, Flow, Mechanism
    from oracle import port
    dev = _dev()
    t = _tables(*shape, tmp_path)
    c, rho = _states(t, 12)
    opts = dict(atol=1e-15, rtol=1e-6, reactor=reactor)
    o = port.integrate(port.MechDesc(t), c.T, c.p, rho, c.Y, 1e-8, opts=port.default_opts(**opts))
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
    m = Mechanism(t)
    flow = Flow(d(c.T), d(c.p), d(rho), d(c.Y))
    cs = ChemistrySource(m, flow, **opts)
    cs.solveUpdate(torch.full((12,), 1e-8, dtype=torch.float64, device=dev), 1.0, counters=True)
    g = {"T": flow.T.cpu().numpy(), "rho": flow.rho.cpu().numpy(), "Y": flow.Y.cpu().numpy()}
    inp = (c.T, c.p, rho, c.Y)
    ref = {k: o[k] for k in ("T", "rho", "Y")}
    check(t, inp, g, ref, 1e-8, opts, f"{shape[0]} species, reactor {reactor}")
    assert (cs.status.cpu().numpy() == 0).all()
    m.close()


@pytest.mark.parametrize("name", ["small", "large"])
def test_properties_rounding_errors(name, request):
    """Properties against extended precision: the root mean square of the relative error in
    units u = 2^-53. A rounding's error is up to u, 0.42 u in the mean square (uniform, and a
    value lies anywhere between two powers of 2). Per value, independent ones adding in
    quadrature: h about 2 beside its largest term (bar 0.65), cp a sum of 5-term polynomials
    (10: 1.4), mu 18 (sqrt T, the power of T, the collision integral, the mixture's sums:
    1.8), kappa another 9 (2.2), D two sums and T^1.5 / p (44: 2.8), times 1 / (1 - x), which
    the species that makes up a cell loses."""
    from openhurricane_b200 import synth
    from openhurricane_b200.chemistry import Mechanism
    dev = _dev()
    t = request.getfixturevalue(name)["tables"]
    L = np.longdouble
    c = synth.dirichlet_cells(t.nsp, 400, seed=11, T_range=(800.0, 2800.0), alpha=0.3)
    T, p, Y, W, e, sg = (np.asarray(a).astype(L) for a in (c.T, c.p, c.Y, t.W[:, None], t.eps_k, t.sigma))
    hi = T[None] >= np.asarray(t.Trange[:, 1])[:, None]
    a = [np.where(hi, t.nasa[:, 1, k][:, None], t.nasa[:, 0, k][:, None]).astype(L) for k in range(7)]
    cp = a[0] + T * (a[1] + T * (a[2] + T * (a[3] + T * a[4])))
    ha = T * (a[0] + T * (a[1] / 2 + T * (a[2] / 3 + T * (a[3] / 4 + T * a[4] / 5)))) + a[5]
    Ru = L(1.380649e-23 * 6.02214076e23 * 1e3)
    X = Y / W
    X /= X.sum(0)
    Ts = T[None] / e[:, None]
    mu = L(2.6693e-6) * np.sqrt(W * T) / (sg[:, None] ** 2 * (L(1.147) * Ts ** L(-0.145) + (Ts + L(0.5)) ** -2))
    num, kap, D = np.zeros_like(T), np.zeros_like(T), np.empty_like(Y)
    for i in range(t.nsp):
        wr = W[i] / W
        w = X[i] * mu[i] / (X * (1 + np.sqrt(mu[i] / mu) * wr ** L(-0.25)) ** 2 / np.sqrt(8 * (1 + wr))).sum(0)
        num += w
        kap += w * (cp[i] + L(1.25) * Ru / W[i])
        Ts = T[None] / np.sqrt(e[i] * e)[:, None]
        s2 = ((sg[i] + sg) / 2)[:, None] ** 2
        q = X * s2 * (Ts ** L(-0.145) + (Ts + L(0.5)) ** -2) * p / (
            L(1.858e-7) * T ** L(1.5) * np.sqrt(1 / W[i] + 1 / W) * L(101325.0))
        D[i] = (1 - X[i]) / (q.sum(0) - q[i])
    m = Mechanism(t)
    g = m.properties(*[torch.tensor(np.ascontiguousarray(v), dtype=torch.float64, device=dev) for v in (c.T, c.p, c.Y)])
    u, bad = 2.0 ** -53, []
    for k, ref, bar in (("ha", ha, 0.65), ("cp", (Y * cp).sum(0), 1.4), ("mu", num, 1.8), ("kappa", kap, 2.2),
                        ("D", D, 2.8)):
        r = (g[k].cpu().numpy().astype(L) - ref) / (np.abs(ref) + (cp * T if k == "ha" else 0.0))
        r = r * (1 - X) if k == "D" else r
        rms = float(np.sqrt((r ** 2).mean()))
        bad = bad + [(k, rms / u)] if rms > bar * u else bad
    m.close()
    assert not bad, bad


@pytest.mark.parametrize("name", ["small", "large"])
def test_rate_constants_and_concentrations_near_underflow(name, request):
    """A fall-off reaction whose high-pressure rate lies below the normal range (its
    reciprocal is needed for the reduced pressure), and concentrations whose products
    underflow unless the large reverse rates of a low temperature come first."""
    import dataclasses
    from openhurricane_b200.chemistry import Mechanism
    from oracle import port, srcimp_oracle
    dev = _dev()
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
    t = request.getfixturevalue(name)["tables"]
    arr, arr0 = t.arr.copy(), t.arr0.copy()
    for r in np.nonzero(t.rate_type >= 2)[0]:
        arr[r] = (1e15, 0.0, 300.0 * (np.log(1e15) + 714.0))       # 1e-310 at 300 K
        arr0[r] = (1e20, 0.0, 0.98 * arr[r, 2])
    for t, T, scale in ((dataclasses.replace(t, arr=arr, arr0=arr0), (299.0, 303.0), 1.0), (t, (55.0, 65.0), 1e-200)):
        c, rho = _states(t, 65)
        c.T[:] = np.linspace(*T, 65)
        rho = rho * scale
        m = Mechanism(t)
        ref = srcimp_oracle.srcimp(t, c.T, c.p, rho, c.Y)
        assert np.isfinite(ref["Ri"]).all() and np.isfinite(ref["diag"]).all()
        args = d(c.T), d(c.p), d(rho), d(c.Y)
        _close(m.source_terms(*args), ref["Ri"], 1e-11, 0, "source")
        Ri, diag = m.source_terms_imp(*args)
        _close(Ri, ref["Ri"], 1e-11, 0, "implicit Ri")
        _close(diag, ref["diag"], 1e-11, 0, "diag")
        conc = rho[None] * c.Y / t.W[:, None]
        f, J = port.rhs_jac(port.MechDesc(t), conc, c.T, c.p)
        gf, gJ = m.rhs_jacobian(d(conc), args[0], args[1])
        _close(gf[:, :t.nsp], f[:, :t.nsp], 1e-11, 1, "f")
        _close(gJ[:, :t.nsp], J[:, :t.nsp], 1e-11, 2, "J")
        m.close()
