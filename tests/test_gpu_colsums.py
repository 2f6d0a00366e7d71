"""GPU tests of column sums on both sides of the line between one cluster and two kernels: rows around the row groups of 8, columns
around the 32- and 128-wide blocks.  Reference in float64; sums of up to 9000 Float32 terms of either sign: 1e-5 of the
largest sum of magnitudes."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


@pytest.mark.parametrize("n", [1, 7, 8, 9, 64, 65, 100, 511, 512, 513])
@pytest.mark.parametrize("cols", [1, 3, 4, 127, 128, 129, 132, 516])
@pytest.mark.parametrize("act", ["identity", "relu", "gelu_tanh"])
def test_bias_gradients(n, cols, act):
    import fluxb200 as F
    from fluxb200 import lib
    ctx, K = F.context(0), 4
    g = torch.Generator(device="cuda").manual_seed(n + cols)
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    W, x, z, dy = new(K, cols), new(n, K), new(n, cols), new(n, cols)
    y = z.relu()
    delta, dW, db = torch.empty(n, cols, device="cuda"), torch.empty_like(W), torch.full((cols + 1,), 7.0, device="cuda")
    lib.call("fb_dense_bwd", ctx.handle, ctx.stream, lib.ACT[act], 0, _p(W), _p(x), _p(y), _p(z), _p(dy), _p(delta), _p(dW), _p(db), None, cols, K, n)
    zz = z.double().requires_grad_()
    f = {"identity": lambda v: v, "relu": torch.relu, "gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[act]
    (f(zz) * dy.double()).sum().backward()
    want = zz.grad
    if act != "identity":
        assert float((delta.double() - want).abs().max()) <= 1e-5 * float(want.abs().max())
    assert float((db[:cols].double() - want.sum(0)).abs().max()) <= 1e-5 * float(want.abs().sum(0).max()) and float(db[cols]) == 7.0
    ref = x.double().T @ want
    assert float((dW.double() - ref).abs().max()) <= 1e-5 * float((x.double().abs().T @ want.abs()).max()) and ctx.device_error() == 0


@pytest.mark.parametrize("d", [1, 5, 40, 132, 1001])
@pytest.mark.parametrize("n", [33, 512, 513, 1025, 2049, 9000])
def test_layernorm_parameter_gradients(d, n):
    import fluxb200 as F
    from fluxb200 import lib
    ctx = F.context(0)
    g = torch.Generator(device="cuda").manual_seed(n + d)
    x, dy = (torch.randn(n, d, generator=g, device="cuda") for _ in range(2))
    mean, rstd = torch.randn(n, generator=g, device="cuda"), torch.rand(n, generator=g, device="cuda") + 0.5
    dg, db = torch.full((d + 1,), 7.0, device="cuda"), torch.full((d + 1,), 7.0, device="cuda")
    one = torch.ones(d, device="cuda")
    lib.call("fb_layernorm_bwd_params", ctx.handle, ctx.stream, _p(x), _p(one), _p(one), _p(mean), _p(rstd), _p(dy), 2.0, _p(dg), _p(db), d, n, 0)
    h = (x.double() - mean.double()[:, None]) * rstd.double()[:, None]
    t = 2.0 * dy.double() * h
    assert float((dg[:d].double() - t.sum(0)).abs().max()) <= 1e-5 * float(t.abs().sum(0).max()) and float(dg[d]) == 7.0
    t = 2.0 * dy.double()
    assert float((db[:d].double() - t.sum(0)).abs().max()) <= 1e-5 * float(t.abs().sum(0).max()) and float(db[d]) == 7.0
