"""GPU tests of the normalisation kernels at the edges of their splits: rows of a warp and of a block, aligned and not, channels
shared by 1 .. 8 CTAs, cached in shared memory or not, and the reverse passes that leave dx out.  Reference: float64 autograd.

Tolerance: sums of up to 2e5 Float32 terms, partly in sequence: 1e-5 of the largest element."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
ACTS = {"identity": lambda v: v, "relu": torch.relu, "gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}


@pytest.fixture(scope="module")
def ctx():
    import fluxb200 as F
    return F.context(0)


def _close(got, ref, name, tol=1e-5):
    err = float((got.double() - ref).abs().max() / ref.abs().max().clamp_min(1e-30))
    assert err < tol, (name, err)


def _p(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


@pytest.mark.parametrize("d", [1, 3, 31, 32, 33, 127, 128, 132, 256, 257, 500, 512, 513, 1000, 1001, 1024, 1025, 1028, 2047, 2048, 2049, 4099, 8191, 8193])
@pytest.mark.parametrize("n,act,shift", [(1, "identity", 0), (9, "gelu_tanh", 0), (700, "relu", 1)])
def test_layernorm_rows(ctx, d, n, act, shift):
    """`shift` floats in front of every array: rows that do not start on 16-byte boundaries whatever d is."""
    from fluxb200 import lib
    g = torch.Generator(device="cuda").manual_seed(d + n)
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, dy = (new(n * d + shift)[shift:].view(n, d) for _ in range(2))
    x = x * 2 + 0.5 if shift == 0 else x
    gamma, beta = new(d) * 0.1 + 1, new(d) * 0.1
    y, dx = (torch.full((n * d + shift,), 7.0, device="cuda")[shift:].view(n, d) for _ in range(2))
    mean, rstd, dg, db, dg2, db2 = (torch.empty(k, device="cuda") for k in (n, n, d, d, d, d))
    a = lib.ACT[act]
    lib.call("fb_layernorm_fwd", ctx.handle, ctx.stream, _p(x), _p(gamma), _p(beta), _p(y), _p(mean), _p(rstd), d, n, 1e-5, a)
    lib.call("fb_layernorm_bwd", ctx.handle, ctx.stream, _p(x), _p(gamma), _p(beta), _p(mean), _p(rstd), _p(dy), _p(dx), _p(dg), _p(db), d, n, a)
    lib.call("fb_layernorm_bwd_params", ctx.handle, ctx.stream, _p(x), _p(gamma), _p(beta), _p(mean), _p(rstd), _p(dy), -1.5, _p(dg2), _p(db2), d, n, a)
    xr, gr, br = (t.double().detach().requires_grad_() for t in (x, gamma, beta))
    z = torch.nn.functional.layer_norm(xr, (d,), gr, br, 1e-5)
    ref = ACTS[act](z)
    if act == "relu":       # an element within rounding of zero may take either side
        dy = torch.where(z.detach().abs() < 1e-5, 0.0, dy.double()).float()
        lib.call("fb_layernorm_bwd", ctx.handle, ctx.stream, _p(x), _p(gamma), _p(beta), _p(mean), _p(rstd), _p(dy), _p(dx), _p(dg), _p(db), d, n, a)
        lib.call("fb_layernorm_bwd_params", ctx.handle, ctx.stream, _p(x), _p(gamma), _p(beta), _p(mean), _p(rstd), _p(dy), -1.5, _p(dg2), _p(db2), d, n, a)
    ref.backward(dy.double())
    _close(y, ref.detach(), "y")
    if d > 1:               # (a row of one element has no gradient, only rounding)
        _close(dx, xr.grad, "dx", 2e-5)
        _close(dg, gr.grad, "dgamma")
        _close(dg2, -1.5 * gr.grad, "dgamma alone")
    _close(db, br.grad, "dbeta")
    _close(db2, -1.5 * br.grad, "dbeta alone")


@pytest.mark.parametrize("s,c,n", [(1, 1, 2), (1, 16, 2), (1, 300, 256), (49, 17, 33), (64, 16, 8), (196, 40, 64), (784, 3, 100), (1024, 8, 128),
                                   (1024, 200, 9), (1022, 5, 31), (1030, 2, 257), (36, 700, 3), (16384, 2, 40), (100000, 1, 3), (4, 3, 70000)])
@pytest.mark.parametrize("act,affine", [("identity", True), ("relu", False), ("gelu_tanh", True)])
def test_batchnorm_channels(ctx, s, c, n, act, affine):
    from fluxb200 import lib
    g = torch.Generator(device="cuda").manual_seed(s + c + n)
    new = lambda *k: torch.randn(*k, generator=g, device="cuda")
    x, dy = new(n, c, s) * 2 + 3, new(n, c, s)
    gamma, beta = (new(c) * 0.1 + 1, new(c) * 0.1) if affine else (None, None)
    rm, rv = new(c), torch.rand(c, generator=g, device="cuda") + 0.5
    rm0, rv0 = rm.clone(), rv.clone()
    y, dx = torch.empty_like(x), torch.empty_like(x)
    mean, rstd, dg, db, dg2, db2 = (torch.empty(c, device="cuda") for _ in range(6))
    a = lib.ACT[act]
    xr = x.double().requires_grad_()
    gr, br = (t.double().requires_grad_() if affine else None for t in (gamma, beta))
    rm64, rv64 = rm.double(), rv.double()
    z = torch.nn.functional.batch_norm(xr, rm64, rv64, gr, br, True, 0.1, 1e-5)
    dy = torch.where(z.detach().abs() < 1e-5, 0.0, dy.double()).float() if act == "relu" else dy
    lib.call("fb_batchnorm_fwd_train", ctx.handle, ctx.stream, _p(x), _p(gamma), _p(beta), _p(rm), _p(rv), _p(y), _p(mean), _p(rstd), s, c, n, 1e-5, 0.1, a, 1)
    lib.call("fb_batchnorm_bwd", ctx.handle, ctx.stream, _p(x), _p(gamma), _p(beta), _p(mean), _p(rstd), _p(dy), _p(dx), _p(dg), _p(db), s, c, n, a)
    lib.call("fb_batchnorm_bwd_params", ctx.handle, ctx.stream, _p(x), _p(gamma), _p(beta), _p(mean), _p(rstd), _p(dy), 0.25, _p(dg2), _p(db2), s, c, n, a)
    ref = ACTS[act](z)
    ref.backward(dy.double())
    _close(y, ref.detach(), "y")
    _close(rm, rm64, "running mean")
    _close(rv, rv64, "running variance")
    if s * n > 2:           # (two values of a channel are +-1 whatever they are)
        _close(dx, xr.grad, "dx", 3e-5)
    if affine:
        scale = float(dy.double().abs().sum(dim=(0, 2)).max())      # sums over a channel cancel
        assert float((dg.double() - gr.grad).abs().max()) < 1e-5 * scale and float((db.double() - br.grad).abs().max()) < 1e-5 * scale
    assert float((dg2 - 0.25 * dg).abs().max()) <= 1e-6 * float(dg.abs().max()) and float((db2 - 0.25 * db).abs().max()) <= 1e-6 * float(db.abs().max())
    lib.call("fb_batchnorm_fwd_infer", ctx.handle, ctx.stream, _p(x), _p(gamma), _p(beta), _p(rm0), _p(rv0), _p(y), s, c, n, 1e-5, a)
    inf = torch.nn.functional.batch_norm(x.double(), rm0.double(), rv0.double(), *(None if t is None else t.double() for t in (gamma, beta)), False, 0.1, 1e-5)
    _close(y, ACTS[act](inf), "inference")
    lib.call("fb_batchnorm_fwd_infer", ctx.handle, ctx.stream, _p(x), _p(gamma), _p(beta), None, None, _p(y), s, c, n, 1e-5, a)
    _close(y, ref.detach(), "inference on batch statistics")


def test_cotangent_known_to_be_a_multiple(ctx):
    """2y, the cotangent of sum(abs2, y), is made when something reads it: next to another use of y, and with the array handed out
    in a second term."""
    import fluxb200 as F
    import numpy as np
    rng = np.random.default_rng(0)
    x = rng.standard_normal((40, 30), dtype=np.float32)
    ln = F.LayerNorm(40)
    xg = F.gpu(x)

    def loss(m, terms):
        y = m(xg)
        out = F.sum_abs2(y)
        for _ in range(terms - 1):
            out = F.add(out, F.sum_abs2(y))
        return out
    one = F.withgradient(lambda m: loss(m, 1), ln)[1][0]["diag"]
    two = F.withgradient(lambda m: loss(m, 2), ln)[1][0]["diag"]
    for k in ("scale", "bias"):
        a, b = F.cpu(one[k]), F.cpu(two[k])
        np.testing.assert_allclose(b, 2 * a, rtol=1e-5, atol=1e-5 * np.abs(a).max())
    y = F.cpu(ln(xg))
    np.testing.assert_allclose(F.cpu(one["bias"]), 2 * y.astype(np.float64).sum(axis=1), rtol=1e-4, atol=1e-4)
