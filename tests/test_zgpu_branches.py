"""The evaluation and integration kernels on the GPU against the CPU oracle on what the
seeded mechanisms do not have: three factors a side and a species three times, irreversible
reactions, Lindemann and three-parameter Troe fall-off, third bodies that are one species or
count one below 1/4, and, where a kernel has a general form for them, species on both
sides, four participants a side and orders that are not the coefficients; every layout of
the warp-per-cell integrator, its build for many cells and autoUpdateJacobian.

Tolerances: those of test_zgpu_evaluation.py for the evaluations, the parity bar and its
one-ulp explanation (parity_util) for the integrations."""
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from test_zgpu_evaluation import _check, _dev, _states, _tables  # noqa: E402

pytestmark = pytest.mark.gpu


def _side(idx, nu, r, species, coef):
    n = len(species)
    idx[r, :n], nu[r, :n] = species, coef
    return n


def _reverse_over_forward(t, r):
    """The largest kr / kf of reaction r over the temperatures of the tests' cells."""
    worst = 1.0
    for T in np.linspace(700.0, 3500.0, 57):
        a = np.where(T >= t.Trange[:, 1, None], t.nasa[:, 1], t.nasa[:, 0]).T
        g = (a[0] * (1 - np.log(T)) - T * (a[1] / 2 + T * (a[2] / 6 + T * (a[3] / 12 + T * a[4] / 20))) + a[5] / T - a[6])
        g = g * t.W / 8314.462618
        dg = sum(v * g[i] for i, v in zip(t.bidx[r, :t.nb[r]], t.bnu[r])) - sum(
            v * g[i] for i, v in zip(t.fidx[r, :t.nf[r]], t.fnu[r]))
        worst = max(worst, float(np.exp(min(dg, 500.0)) * (8314.462618 * T / 101325.0) ** t.sum_stoi[r]))
    return worst


def odd_tables(t, general, alone=True):
    """Copies of the tables with their first reactions replaced and, where `alone`, the others'
    rate constants zero. The species do not balance elements, so a rate constant is divided
    by what its reverse would exceed it by."""
    t = dataclasses.replace(t, **{k: getattr(t, k).copy() for k in
                                  ("rate_type", "reversible", "arr", "arr0", "troe", "eff", "nf", "nb", "fidx", "bidx",
                                   "fnu", "bnu", "ford", "bord", "sum_stoi")})
    s = t.nsp
    sides = [([0, 1, 2], [1, 1, 1], [3, 4], [1, 1]),            # three factors, one mole less
             ([1, 2], [2, 1], [0, 3], [1, 2]),                  # repeated factors on both sides
             ([4], [3], [0, 1, 2], [1, 1, 1]),                  # a species three times
             ([0, s - 1], [1, 1], [1, 3], [1, 1]),              # irreversible
             ([2, 3], [1, 1], [s - 1], [1]),                    # third body: one species only
             ([3], [1], [0, s - 1], [1, 1]),                    # third body: one efficiency of 0.1
             ([1, 3], [1, 1], [4], [1]),                        # Lindemann
             ([0, 2], [1, 1], [s - 1], [1]),                    # Troe, three parameters
             ([s - 1], [2], [3, 4], [1, 1])]                    # irreversible third body
    if general:
        sides += [([0, 1], [1, 2], [1, 2], [1, 1]),             # a species on both sides
                  ([0, 1, 2, 3], [1, 1, 1, 1], [4], [1]),       # four participants
                  ([2, 4], [1, 1], [0], [1])]                   # orders 0.5 and 1.7
    for r, (f, fn, b, bn) in enumerate(sides):
        t.nf[r] = _side(t.fidx, t.fnu, r, f, fn)
        t.nb[r] = _side(t.bidx, t.bnu, r, b, bn)
        t.ford[r], t.bord[r] = t.fnu[r], t.bnu[r]
        t.sum_stoi[r] = sum(bn) - sum(fn)
        t.rate_type[r], t.reversible[r], t.eff[r] = 0, 1, 1.0
        order = sum(fn)
        t.arr[r] = (1e9 * 100.0 ** (order - 2), 0.3, 2000.0 + 300.0 * r)
        if r not in (3, 8):                                     # the irreversible ones
            t.arr[r, 0] /= _reverse_over_forward(t, r)
    t.reversible[[3, 8]] = 0
    t.rate_type[[4, 5, 8]] = 1
    t.eff[4] = 0.0
    t.eff[4, 1] = 1.0
    t.eff[5, 2] = 0.1
    t.eff[8, :3] = (2.5, 0.0, 12.0)
    t.rate_type[6], t.rate_type[7] = 2, 3
    for r in (6, 7):
        t.arr0[r] = (300.0 * t.arr[r, 0], -0.8, 500.0)
    t.troe[7] = (0.6, 150.0, 1800.0, 0.0)
    if general:
        t.ford[11, :2] = (0.5, 1.7)
    if alone:
        t.arr[len(sides):, 0] = t.arr0[len(sides):, 0] = 0.0
    return t


def only(t, r):
    """The tables with every rate constant but reaction r's zero."""
    arr, arr0 = t.arr.copy(), t.arr0.copy()
    rest = np.arange(t.nrc) != r
    arr[rest, 0] = arr0[rest, 0] = 0.0
    return dataclasses.replace(t, arr=arr, arr0=arr0)


SIZES = [(7, 14, 2, 1), (10, 20, 4, 1), (15, 45, 8, 3), (20, 60, 10, 4), (33, 120, 20, 6), (56, 300, 50, 12),
         (63, 400, 60, 20)]


@pytest.mark.parametrize("general", [False, True], ids=["direct", "general"])
@pytest.mark.parametrize("shape", SIZES, ids=lambda s: f"{s[0]}sp")
def test_evaluations(shape, general, tmp_path):
    base = _tables(*shape, tmp_path)
    t = odd_tables(base, general)
    for r in range(12 if general else 9):
        _check(only(t, r), 5)                # a row's tolerance is of its largest element
    _check(t, 33, cold=True)
    _check(odd_tables(base, general, alone=False), 33)


# some hundred Newton iterations a cell; a cell that needed more would be flagged
OPTS = dict(atol=1e-15, rtol=1e-6, max_newton_total=100000)


def slower(t):
    """The tables with every rate 1e-4 of what it was: the random mechanisms' cells change
    by hundreds of degrees within 1e-8 s all the same."""
    arr, arr0 = t.arr.copy(), t.arr0.copy()
    arr[:, 0] *= 1e-4
    arr0[:, 0] *= 1e-4
    return dataclasses.replace(t, arr=arr, arr0=arr0)


def _integrate(t, c, rho, dt, opts):
    from openhurricane_b200.chemistry import ChemistrySource, Flow, Mechanism
    dev, n = _dev(), c.T.shape[0]
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
    m = Mechanism(t)
    flow = Flow(d(c.T), d(c.p), d(rho), d(c.Y))
    cs = ChemistrySource(m, flow, **opts)
    cs.solveUpdate(torch.full((n,), dt, dtype=torch.float64, device=dev), 1.0, counters=True)
    g = {"T": flow.T.cpu().numpy(), "rho": flow.rho.cpu().numpy(), "Y": flow.Y.cpu().numpy()}
    status = cs.status.cpu().numpy()
    m.close()
    return g, status, cs.last_counters


def _against_oracle(t, n, dt, opts, what):
    from oracle import port
    from parity_util import check
    c, rho = _states(t, n)
    o = port.integrate(port.MechDesc(t), c.T, c.p, rho, c.Y, dt, opts=port.default_opts(**opts))
    g, status, counters = _integrate(t, c, rho, dt, opts)
    check(t, (c.T, c.p, rho, c.Y), g, {k: o[k] for k in ("T", "rho", "Y")}, dt, opts, what)
    assert (status == 0).all()
    return counters


@pytest.mark.parametrize("reactor", [0, 1])
@pytest.mark.parametrize("general", [False, True], ids=["direct", "general"])
@pytest.mark.parametrize("shape", SIZES[:5], ids=lambda s: f"{s[0]}sp")
def test_integrations(shape, general, reactor, tmp_path):
    t = odd_tables(_tables(*shape, tmp_path), general)
    _against_oracle(t, 12, 1e-8, dict(OPTS, reactor=reactor), f"{shape} {general} {reactor}")


@pytest.mark.parametrize("reactor", [0, 1])
@pytest.mark.parametrize("shape", [(7, 14, 2, 1), (9, 21, 3, 1), (10, 20, 4, 1), (15, 45, 8, 3)],
                         ids=lambda s: f"{s[0]}sp")
@pytest.mark.parametrize("every", [0, 2, 10])
def test_layouts_and_auto_update_jacobian(shape, reactor, every, tmp_path):
    """every: Newton iterations between Jacobians, 0: a new one in each. With a Jacobian that
    stays, Newton converges in more iterations to the same answer."""
    t = slower(_tables(*shape, tmp_path))
    opts = dict(OPTS, reactor=reactor)
    if every:
        opts.update(auto_update_jacobian=1, step_to_update_jac=every)
    n = _against_oracle(t, 16, 1e-8, opts, f"{shape} {reactor} {every}")
    assert n["n_lu"] == n["n_jac"] and n["n_newton"] + 16 >= n["n_rhs"]
    assert (n["n_jac"] < n["n_newton"]) == bool(every)


@pytest.mark.parametrize("reactor", [0, 1])
@pytest.mark.parametrize("shape", [(9, 21, 3, 1), (12, 26, 4, 2)], ids=lambda s: f"{s[0]}sp")
def test_build_for_many_cells(shape, reactor, tmp_path):
    """From 8 cells for each warp of two blocks per SM (18,944 on 148 SMs) kernel 6 is another
    build. 200 states, each a hundred times: every copy gives the same answer, and a sample
    of them the oracle's."""
    from oracle import port
    from parity_util import check
    t = slower(_tables(*shape, tmp_path))
    c, rho = _states(t, 200)
    opts = dict(OPTS, reactor=reactor)
    many = dataclasses.replace(c, T=np.tile(c.T, 100), p=np.tile(c.p, 100), Y=np.tile(c.Y, 100))
    g, status, _ = _integrate(t, many, np.tile(rho, 100), 1e-8, opts)
    assert (status == 0).all()
    first = {k: v[..., :200] for k, v in g.items()}
    for k, v in g.items():
        assert np.array_equal(v, np.tile(first[k], 100)), k
    s = slice(0, 40)
    o = port.integrate(port.MechDesc(t), c.T[s], c.p[s], rho[s], np.ascontiguousarray(c.Y[:, s]), 1e-8,
                       opts=port.default_opts(**opts))
    check(t, (c.T[s], c.p[s], rho[s], np.ascontiguousarray(c.Y[:, s])), {k: v[..., s] for k, v in first.items()},
          {k: o[k] for k in ("T", "rho", "Y")}, 1e-8, opts, f"{shape} {reactor}")


def test_a_kept_jacobian_shortens_the_iteration(tmp_path):
    """One cell of 15 species, where the time is that of its Newton iterations in a chain: with
    the factors kept for up to ten of them an iteration takes at most 0.9 of the time it
    takes with a Jacobian each. (Forming the matrix and eliminating again took 0.96.)"""
    from openhurricane_b200.chemistry import ChemistrySource, Flow, Mechanism
    dev = _dev()
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
    t = slower(_tables(15, 45, 8, 3, tmp_path))
    c, rho = _states(t, 1)
    m = Mechanism(t)
    dt = torch.full((1,), 1e-7, dtype=torch.float64, device=dev)
    per = {}
    for auto in (0, 1):
        best = np.inf
        for _ in range(4):
            cs = ChemistrySource(m, Flow(d(c.T), d(c.p), d(rho), d(c.Y)), auto_update_jacobian=auto,
                                 step_to_update_jac=10, **OPTS)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            cs.solveUpdate(dt, 1.0)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) / int(cs.cost[0]))
        per[auto] = best
    assert per[1] <= 0.9 * per[0], per
    m.close()


def test_more_cells_do_not_take_a_build_that_does_not_fit_twice(tmp_path):
    """The build for two blocks an SM pays where shared memory holds two. With 15 species and
    45 reactions it holds one: a ninth more cells (18,000 and 20,000 lie on both sides of
    the line for 148 SMs) may take a fifth more time. (The other build took a third more.)"""
    from openhurricane_b200.chemistry import ChemistrySource, Flow, Mechanism
    dev = _dev()
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
    t = slower(_tables(15, 45, 8, 3, tmp_path))
    c, rho = _states(t, 200)
    m, took = Mechanism(t), {}
    for n in (90, 100):
        state = [np.tile(a, n) for a in (c.T, c.p, rho, c.Y)]
        took[n] = np.inf
        for _ in range(2):
            cs = ChemistrySource(m, Flow(*[d(a) for a in state]), **OPTS)
            dt = torch.full((200 * n,), 1e-8, dtype=torch.float64, device=dev)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            cs.solveUpdate(dt, 1.0)
            b.record()
            torch.cuda.synchronize()
            took[n] = min(took[n], a.elapsed_time(b))
    assert took[100] <= 1.2 * took[90], took
    m.close()
