"""GPU tests of bf16 Dense layers at the edges of the GEMM's 64-column stores and of the activation's reverse pass.  References are computed in
float64 from the same rounded arrays; a BFloat16 result may be off by one rounding (2^-8 of the value) where a Float32
result lies within 1e-5 of a tie, so these compare with 2^-8 of the element plus 1e-5 of the largest."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
ACTS = {"identity": lambda v: v, "relu": torch.relu, "gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}
BF = torch.bfloat16


@pytest.fixture(scope="module")
def ctx():
    import fluxb200 as F
    return F.context(0)


def _p(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def _close(got, ref, name, tol=1e-5):
    lim = tol * ref.abs().max() + (2.0 ** -8 * ref.abs() if got.dtype == BF else 0.0)
    assert bool(((got.double() - ref).abs() <= lim).all()), (name, float((got.double() - ref).abs().max()), float(ref.abs().max()))


@pytest.mark.parametrize("out_dim,in_dim,n", [(8, 16, 1), (64, 64, 130), (128, 72, 129), (264, 136, 300), (520, 256, 513), (1000, 512, 1024),
                                              (1024, 1024, 4096), (2048, 512, 2050)])
@pytest.mark.parametrize("act", ["identity", "relu", "tanh", "gelu_tanh"])
def test_dense_bf16(ctx, out_dim, in_dim, n, act):
    """Sums of up to 4096 products in Float32 (truncated as they are added: 2e-5 of the largest) around BFloat16 roundings."""
    from fluxb200 import lib
    g = torch.Generator(device="cuda").manual_seed(out_dim + n)
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    W, b, x, dy = (new(in_dim, out_dim) / in_dim ** 0.5).to(BF), new(out_dim).to(BF), new(n, in_dim).to(BF), new(n, out_dim).to(BF)
    y, z, delta = (torch.empty(n, out_dim, device="cuda", dtype=BF) for _ in range(3))
    dW, db, dx = torch.empty_like(W), torch.empty_like(b), torch.empty_like(x)
    a = lib.ACT[act]
    lib.call("fb_dense_fwd_bf16", ctx.handle, ctx.stream, a, _p(W), _p(b), _p(x), _p(y), _p(z), out_dim, in_dim, n)
    zr = x.double() @ W.double() + b.double()
    f = {**ACTS, "tanh": torch.tanh}[act]
    _close(z, zr, "z", 2e-5)
    _close(y, f(zr), "y", 2e-5)
    lib.call("fb_dense_bwd_bf16", ctx.handle, ctx.stream, a, _p(W), _p(x), _p(y), _p(z), _p(dy), _p(delta), _p(dW), _p(db), _p(dx), out_dim, in_dim, n)
    zz = z.double().requires_grad_()
    if act in ("relu", "tanh"):
        want = dy.double() * ((y > 0).double() if act == "relu" else 1 - y.double() ** 2)
    else:
        f(zz).backward(dy.double())
        want = zz.grad
    if act != "identity":
        _close(delta, want, "delta", 2e-5)
    d = delta.double() if act != "identity" else dy.double()
    _close(db, d.sum(0), "db", 2e-5)
    _close(dW, x.double().T @ d, "dW", 4e-5)
    _close(dx, d @ W.double().T, "dx", 4e-5)
    assert ctx.device_error() == 0
