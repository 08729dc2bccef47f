"""The network's inference kernel and the ensemble kernel on the GPU: the
fused forward pass at the edges of its tiles and shapes (and the layer-by-layer
one just past them) against the same network in float64 on the operands the
kernel multiplies, the ensemble's mean and spread against the same formulas."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _dev():
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch.device("cuda:0")


def _reference(theta, shapes, X, wrong=None):
    """float64, with the input, the weights and every activation rounded to BF16 as the
    kernels round them; also the expected square of the kernels' distance from it. That has
    two sources, which add in quadrature over the products of a layer: float32 accumulation
    (a few 2^-24 of the sum of magnitudes) and activations next to a boundary of BF16, which
    round the other way: with an error s before the rounding that is a step u = 2^-8 |h| in
    0.8 s / u of the cases. `wrong`: the same network with a mistake in it."""
    bf = lambda a: torch.as_tensor(a, dtype=torch.float32).to(torch.bfloat16).double()
    h, var, off = bf(X), 0.0, 0
    for l, (o, i) in enumerate(shapes):
        W = bf(theta[off:off + o * i].reshape(o, i))
        b = torch.as_tensor(theta[off + o * i:off + o * i + o]).double()
        off += o * i + o
        last = l + 1 == len(shapes)
        carried = var @ (W ** 2).T if l else 0.0
        s2 = carried + ((h.abs() @ W.abs().T + b.abs()) * 2.0 ** -23) ** 2
        if wrong == "K block" and last:
            W = torch.cat([torch.zeros_like(W[:, :16]), W[:, 16:]], 1)
        h = h @ W.T + (0.0 if wrong == "bias" else b)
        var = s2
        if not last:
            h = torch.relu(h) if wrong == "ReLU" else torch.nn.functional.gelu(h)
            s = 1.13 * s2.sqrt() + 1e-7              # |gelu'| < 1.13, the error of gelu_f
            var = 0.8 * s * h.abs() * 2.0 ** -8 + s ** 2
            h = bf(h.float())
    return (torch.zeros_like(h) if wrong == "zero" else h), var


def test_gelu_against_float64():
    """The epilogues' GELU of exact float32 arguments (a product with zeros, the arguments
    as the bias): rounding of the result, a dozen float roundings of |z| Q(|z|) and the
    fit's 5e-9; in the negative tail, where the value itself is small, the fit's 5e-5 of it
    and the rounding of the exponent z^2 / 2."""
    from openhurricane_b200.surrogate import gemm_bf16
    dev = _dev()
    rng = np.random.default_rng(0)
    z = np.concatenate([rng.normal(size=200000), rng.uniform(-8, 8, 200000), np.linspace(-8, 8, 62141),
                        [0.0, -0.0, 1e-30, 5e-324, 100.0, 1e30, 3e38]]).astype(np.float32)
    z = np.concatenate([z, np.full(-len(z) % 32, 1.0, np.float32)])
    A = torch.zeros(128, 64, dtype=torch.bfloat16, device=dev)
    B = torch.zeros(len(z), 64, dtype=torch.bfloat16, device=dev)
    got = gemm_bf16(A, B, torch.tensor(z, device=dev), act=1)[0].cpu().double().numpy()
    x = z.astype(np.float64)
    tail = 0.5 * torch.special.erfc(torch.tensor(np.abs(x) / np.sqrt(2.0))).numpy() * np.abs(x)
    ref = np.maximum(x, 0.0) - tail
    assert (np.abs(got - ref) <= 2.0 ** -24 * np.abs(ref) + 12 * 2.0 ** -24 * tail + 5e-9).all()
    low = x < -3.0
    assert (np.abs(got - ref)[low] <= (5e-5 + 2.0 ** -22 * (12.0 + x[low] ** 2)) * -ref[low]).all()
    v = torch.tensor([np.inf, -np.inf, np.nan] + [1.0] * 29, dtype=torch.float32, device=dev)
    got = gemm_bf16(A, B[:32], v, act=1)[0].cpu().numpy()
    assert got[0] == np.inf and np.isnan(got[1]) and np.isnan(got[2]) and np.isfinite(got[3:]).all()


@pytest.mark.parametrize("shape", [(1, 1, 1, 64), (12, 10, 3, 256), (56, 54, 2, 256), (64, 64, 1, 128),
                                   (65, 65, 2, 192), (256, 256, 1, 256), (12, 10, 2, 320)])
@pytest.mark.parametrize("B", [1, 127, 128, 129, 2000])
def test_forward_matches_float64_on_rounded_operands(shape, B):
    from openhurricane_b200.surrogate import MLP
    dev = _dev()
    n_in, n_out, nh, w = shape
    net = MLP(n_in, n_out, nh, w, max_batch=1024, seed=5)
    X = np.random.default_rng(B).normal(size=(B, n_in)).astype(np.float32)
    out = net.forward(torch.tensor(X, device=dev)).cpu().double()
    args = net.get_params(), net.shapes(), X
    ref, var = _reference(*args)
    assert out.shape == ref.shape
    rms = lambda d: float((d ** 2).mean().sqrt())
    bar = 6.0 * float(var.mean().sqrt())
    assert rms(out - ref) <= bar, (rms(out - ref), bar)
    if B >= 127:
        # the bar tells a missing bias, K slice or activation from rounding
        for wrong in ("zero", "bias", "K block", "ReLU"):
            assert rms(_reference(*args, wrong)[0] - ref) > 10 * bar, wrong


@pytest.mark.parametrize("n,n_out,n_nets", [(1, 1, 1), (257, 10, 2), (4096, 54, 4), (1000, 7, 3)])
def test_ensemble_matches_its_formulas(n, n_out, n_nets):
    import ctypes as C
    from openhurricane_b200 import _capi
    dev = _dev()
    rng = np.random.default_rng(n)
    P = rng.normal(size=(n_nets, n, n_out)).astype(np.float32)
    if n > 1:
        P[n_nets - 1, n // 2, n_out - 1] = np.nan
        P[0, n // 3, 0] = np.inf
        P[:, 0, 0] = -np.inf
    scale = rng.uniform(0.5, 2.0, n_out)
    p, s = torch.tensor(P, device=dev), torch.tensor(scale, device=dev)
    mean = torch.empty(n, n_out, dtype=torch.float32, device=dev)
    spread = torch.empty(n, dtype=torch.float32, device=dev)
    vp = lambda t: C.c_void_p(t.data_ptr())
    _capi.check(_capi.load().hc_surrogate_ensemble(n, n_out, n_nets, vp(p), vp(s), 50.0, 1e-2, vp(mean), vp(spread),
                                                   C.c_void_p(torch.cuda.current_stream().cuda_stream)),
                "hc_surrogate_ensemble")
    with np.errstate(invalid="ignore"):
        Q = P.astype(np.float64)
        m = Q.mean(axis=0)
        d = (Q.max(axis=0) - Q.min(axis=0)) * scale / np.where(np.arange(n_out) == 0, 50.0, 1e-2)
        sp = d.max(axis=1)                           # NaN where a prediction is NaN
    # at most n_nets + 1 float32 roundings of values up to the largest magnitude
    tol = (n_nets + 1) * 2.0 ** -23 * np.nanmax(np.where(np.isfinite(Q), np.abs(Q), 0.0))
    got = mean.cpu().numpy()
    np.testing.assert_array_equal(np.isnan(got), np.isnan(m))
    np.testing.assert_allclose(got, m, rtol=0.0, atol=tol)
    np.testing.assert_allclose(spread.cpu().numpy(), sp, rtol=4 * 2.0 ** -23, atol=1e-4)


def test_predict_takes_the_scales_of_any_form(small):
    """out_std as float32, one number or every other element of a tensor gives what the
    same values as consecutive doubles give (the kernel reads those); a scale on another
    device and networks of other widths are refused."""
    from openhurricane_b200.chemistry import Mechanism
    from openhurricane_b200.surrogate import MLP, Surrogate
    dev = _dev()
    sur = Surrogate(Mechanism(small["tables"]), n_hidden=1, width=64, max_batch=256, seed=1)
    X = torch.randn(100, sur.n_in, device=dev)
    base = torch.linspace(0.5, 2.0, sur.n_out, device=dev).float()
    spaced = torch.full((sur.n_out, 2), 7.0, dtype=torch.float64, device=dev)
    spaced[:, 0] = base.double()
    sur.out_std = base.double()
    mean, spread = sur.predict(X)
    for form in (base, spaced[:, 0]):
        sur.out_std = form
        m, s = sur.predict(X)
        assert torch.equal(m, mean) and torch.equal(s, spread)
    sur.out_std = torch.full((sur.n_out,), 0.25, dtype=torch.float64, device=dev)
    _, spread = sur.predict(X)
    sur.out_std = torch.tensor([0.25], dtype=torch.float64, device=dev)
    assert torch.equal(sur.predict(X)[1], spread)
    sur.out_std = base.double().cpu()
    with pytest.raises(ValueError):
        sur.predict(X)
    sur.out_std = base.double()
    sur.nets[1] = MLP(sur.n_in, sur.n_out + 3, 1, 64, max_batch=256)
    with pytest.raises(ValueError):
        sur.predict(X)
