"""GPU tests of the parameter gradients of LayerNorm / BatchNorm where the cotangent is a factor times the layer's own output (sum(abs2, y)):
made from x again, it has the bits of the stored output, so the gradients have those of the general path."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ACTS = ["identity", "relu", "gelu", "sigmoid"]


def _new(g, n, offset=0, scale=1.0, shift=0.0):
    return (torch.randn(n + offset, generator=g, device="cuda") * scale + shift)[offset:]


@pytest.mark.parametrize("act", ACTS)
@pytest.mark.parametrize("s,c,n,offset", [(1024, 256, 16, 0), (49, 33, 20, 0), (1, 17, 300, 0), (64, 5, 3, 1), (25600, 3, 2, 0), (196, 512, 2, 0), (1, 1, 2, 0)])
def test_batchnorm(act, s, c, n, offset):
    import fluxb200 as F
    from fluxb200 import lib
    ctx, g = F.context(0), torch.Generator(device="cuda").manual_seed(s)
    x, ga, be = _new(g, s * c * n, offset, 2.0, 0.5), _new(g, c, 0, 0.1, 1.0), _new(g, c, 0, 0.5)
    y, mean, rstd = torch.empty_like(x), torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    a, p = lib.ACT[act], lambda t: t.data_ptr()
    lib.call("fb_batchnorm_fwd_train", ctx.handle, ctx.stream, p(x), p(ga), p(be), None, None, p(y), p(mean), p(rstd), s, c, n, 1e-5, 0.1, a, 0)
    res = [torch.empty(c, device="cuda") for _ in range(4)]
    lib.call("fb_batchnorm_bwd_params", ctx.handle, ctx.stream, p(x), p(ga), p(be), p(mean), p(rstd), p(y), 2.0, p(res[0]), p(res[1]), s, c, n, a)
    lib.call("fb_batchnorm_bwd_params_own", ctx.handle, ctx.stream, p(x), p(ga), p(be), p(mean), p(rstd), 2.0, p(res[2]), p(res[3]), s, c, n, a)
    assert ctx.device_error() == 0 and torch.equal(res[0], res[2]) and torch.equal(res[1], res[3])


@pytest.mark.parametrize("act", ACTS)
@pytest.mark.parametrize("d,n,offset", [(1001, 3000, 0), (256, 7, 0), (32, 1, 0), (4096, 50, 0), (8192, 3, 0), (100, 999, 1), (1, 5, 0), (9000, 4, 0)])
def test_layernorm(act, d, n, offset):
    import fluxb200 as F
    from fluxb200 import lib
    ctx, g = F.context(0), torch.Generator(device="cuda").manual_seed(d)
    x, ga, be = _new(g, d * n, offset, 2.0, 0.5), _new(g, d, 0, 0.1, 1.0), _new(g, d, 0, 0.5)
    y, mean, rstd = torch.empty_like(x), torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    a, p = lib.ACT[act], lambda t: t.data_ptr()
    lib.call("fb_layernorm_fwd", ctx.handle, ctx.stream, p(x), p(ga), p(be), p(y), p(mean), p(rstd), d, n, 1e-5, a)
    res = [torch.empty(d, device="cuda") for _ in range(4)]
    lib.call("fb_layernorm_bwd_params", ctx.handle, ctx.stream, p(x), p(ga), p(be), p(mean), p(rstd), p(y), 2.0, p(res[0]), p(res[1]), d, n, a)
    lib.call("fb_layernorm_bwd_params_own", ctx.handle, ctx.stream, p(x), p(ga), p(be), p(mean), p(rstd), 2.0, p(res[2]), p(res[3]), d, n, a)
    assert torch.equal(res[0], res[2]) and torch.equal(res[1], res[3])


@pytest.mark.parametrize("kind", ["layer", "batch"])
def test_which_cotangents_take_it(kind, monkeypatch):
    """A factor times y itself; not a sum of two cotangents, a factor times another array, nor a cotangent that somebody has read."""
    import fluxb200 as F
    from fluxb200 import core, lib
    g = torch.Generator(device="cuda").manual_seed(0)
    m = F.LayerNorm(24) if kind == "layer" else F.BatchNorm(24)
    x = F.B200Array(_new(g, 24 * 10), (24, 10))
    other = F.B200Array(_new(g, 24 * 10), (24, 10))
    calls, real = [], lib.call
    monkeypatch.setattr(lib, "call", lambda name, *a: calls.append(name) or real(name, *a))
    general, own = f"fb_{kind}norm_bwd_params", f"fb_{kind}norm_bwd_params_own"

    def grad(f, entry):
        del calls[:]
        res = _arrays(F.withgradient(f, m)[1])
        assert [c for c in calls if "norm_bwd" in c] == [entry], calls
        return res
    one = grad(lambda m: F.sum_abs2(m(x)), own)
    both = grad(lambda m: F.sum_abs2(F.add(m(x), other)), general)
    read = core.is_scaled
    monkeypatch.setattr(core, "is_scaled", lambda g, y: (g.t, read(g, y))[1])   # (the cotangent's memory has been asked for)
    import fluxb200.layers as layers
    monkeypatch.setattr(layers, "is_scaled", core.is_scaled)
    seen = grad(lambda m: F.sum_abs2(m(x)), general)
    assert all(torch.equal(a, b) for a, b in zip(seen, one))
    h = x.t.double().view(10, 24)
    h = (h - h.mean(1, keepdim=True)) / (h.var(1, unbiased=False, keepdim=True) + 1e-5).sqrt() if kind == "layer" else \
        (h - h.mean(0)) / (h.var(0, unbiased=False) + 1e-5).sqrt()
    o = other.t.double().view(10, 24)
    for got, dy in ((one, 2 * h), (both, 2 * (h + o))):
        want = sorted([(dy * h).sum(0), dy.sum(0)], key=lambda t: float(t.norm()))
        got = sorted(got, key=lambda t: float(t.double().norm()))
        for a, b in zip(got, want):
            assert float((a.double() - b).abs().max()) < 1e-5 * float(dy.abs().sum(0).max())


def _arrays(v):
    import fluxb200 as F
    if isinstance(v, F.B200Array):
        return [v.t]
    if isinstance(v, dict):
        v = list(v.values())
    return [t for x in v for t in _arrays(x)] if isinstance(v, (list, tuple)) else []
