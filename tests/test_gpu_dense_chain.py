"""GPU tests of a Chain of Dense layers for a few columns in one launch: slices of 4 to 128 outputs, outputs that fill some of the 16
CTAs only, rows that are not 16-byte aligned, several stages of weights, 1 to 28 columns, and the calls that are left to the layers.

Tolerance: Float32 sums of up to 1000 products in 16 parts, layer after layer: 3e-6 of the result's norm (sums of random signs come
to about 2e-7)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [([784, 512, 512, 10], 1), ([784, 512, 512, 10], 28), ([5, 3, 2], 1), ([64, 65, 63, 7], 3), ([300, 501, 333, 9], 9), ([16, 1025, 1], 2), ([16, 1000, 2], 5),
          ([200, 64, 1024, 17], 4), ([1000, 128, 60], 27), ([33] * 9, 6), ([7, 2000, 4], 1)]


def _chain(F, dims, act, g, offset=0, bias=True):
    def array(*size):
        n = 1
        for s in size:
            n *= s
        return F.B200Array((torch.randn(n + offset, generator=g, device="cuda") / size[-1] ** 0.5)[offset:], size)
    return F.Chain(*[F.Dense(array(o, i), array(o) if bias else False, act if k + 2 < len(dims) else "identity")
                     for k, (i, o) in enumerate(zip(dims, dims[1:]))])


def _reference(F, m, x, n):
    f = {"relu": lambda t: t.clamp(min=0), "identity": lambda t: t, "tanh": torch.tanh, "sigmoid": torch.sigmoid,
         "gelu": lambda t: torch.nn.functional.gelu(t, approximate="tanh")}
    h = x.t.double().view(n, -1)
    for l in m.layers:
        h = h @ l.weight.t.double().view(l.weight.size[1], l.weight.size[0]) + (0 if l.bias is False else l.bias.t.double())
        h = f[l.σ](h)
    return h


@pytest.mark.parametrize("dims,n", SHAPES)
@pytest.mark.parametrize("act,offset,bias", [("relu", 0, True), ("gelu", 1, True), ("tanh", 0, False), ("sigmoid", 2, True)])
def test_chain(dims, n, act, offset, bias):
    import fluxb200 as F
    from fluxb200 import layers
    g = torch.Generator(device="cuda").manual_seed(n)
    m = _chain(F, dims, act, g, offset, bias)
    x = F.B200Array(torch.randn(n * dims[0], generator=g, device="cuda"), (dims[0], n))
    assert layers._dense_chain(m.layers, x) is not None
    y, ref = m(x), _reference(F, m, x, n)
    assert y.size == (dims[-1], n) and F.context(0).device_error() == 0
    err = float((y.t.double().view(n, -1) - ref).norm() / ref.norm())
    assert err < 3e-6, err
    assert torch.equal(m(x).t, y.t)


def test_what_is_left_to_the_layers():
    import fluxb200 as F
    from fluxb200 import layers
    g = torch.Generator(device="cuda").manual_seed(0)
    one = lambda dims, n: layers._dense_chain(_chain(F, dims, "relu", g).layers, F.B200Array(torch.randn(n * dims[0], device="cuda"), (dims[0], n)))
    assert one([64, 64, 8], 28) is not None and one([64, 64, 8], 29) is None
    assert one([2048, 2048, 2048], 1) is None and one([64, 2049, 4], 1) is None and one([64] * 10, 1) is None
    m = _chain(F, [64, 32, 8], "relu", g)
    with pytest.raises(F.DimensionMismatch):
        m(F.B200Array(torch.randn(65, device="cuda"), (65, 1)))
    v = m(F.B200Array(torch.randn(64, device="cuda"), (64,)))
    assert v.size == (8,)
    low = F.bf16(_chain(F, [64, 32, 8], "relu", g))
    assert layers._dense_chain(low.layers, F.B200Array(torch.randn(64, device="cuda"), (64, 1))) is None


def test_values_that_are_not_finite():
    import fluxb200 as F
    g = torch.Generator(device="cuda").manual_seed(0)
    m = _chain(F, [70, 50, 6], "identity", g)
    x = torch.randn(3 * 70, generator=g, device="cuda")
    x[75] = float("inf")
    x = F.B200Array(x, (70, 3))
    y, ref = m(x).t.view(3, 6), _reference(F, m, x, 3)
    assert torch.equal(torch.isfinite(y), torch.isfinite(ref)) and torch.equal(torch.isnan(y), torch.isnan(ref))


def test_captured_and_beside_another_stream():
    import fluxb200 as F
    g = torch.Generator(device="cuda").manual_seed(1)
    m = _chain(F, [784, 512, 512, 10], "relu", g)
    xs = [F.B200Array(torch.randn(784, generator=g, device="cuda"), (784, 1)) for _ in range(2)]
    want = [m(x).t.clone() for x in xs]
    torch.cuda.synchronize()
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph):
        y = m(xs[0])
    for _ in range(3):
        y.t.zero_()
        graph.replay()
        with torch.cuda.stream(side):
            z = m(xs[1])
        torch.cuda.synchronize()
        assert torch.equal(y.t, want[0]) and torch.equal(z.t, want[1])


@pytest.mark.parametrize("size", [(), (65,), (65, 1), (65, 40), (65, 1, 1), (1, 64)])
def test_arrays_of_other_shapes_are_refused_by_the_first_layer(size):
    import fluxb200 as F
    m = _chain(F, [64, 32, 8], "relu", torch.Generator(device="cuda").manual_seed(0))
    n = 1
    for s in size:
        n *= s
    x = F.B200Array(torch.randn(n, device="cuda"), size)
    with pytest.raises(F.DimensionMismatch) as chain:
        m(x)
    with pytest.raises(F.DimensionMismatch) as layer:
        m.layers[0](x)
    assert str(chain.value) == str(layer.value)


def test_large_weights_are_not_asked_about(monkeypatch):
    """The entry point refuses them; a call on a few columns of a large model does not get that far.  (The line: its own, for one column.)"""
    import fluxb200 as F
    from fluxb200 import layers, lib
    asked = []
    real = lib.supported
    monkeypatch.setattr(lib, "supported", lambda name, *a: asked.append(name) or real(name, *a))
    g = torch.Generator(device="cuda").manual_seed(0)
    x = lambda d: F.B200Array(torch.randn(d, device="cuda"), (d, 1))
    for dims, taken in (([1024, 512, 512], True), ([1024, 512, 1024], True), ([1024, 512, 1025], False), ([2048, 2048, 8], False), ([8, 2048, 2048], False), ([1024, 512, 1024, 513], False)):
        del asked[:]
        y = layers._dense_chain(_chain(F, dims, "relu", g).layers, x(dims[0]))
        assert (y is not None) == taken and asked == (["fb_dense_chain_fwd"] if taken else [])


def test_named_entry_points_are_timed(monkeypatch):
    """A call of several layers in one launch is seen where entry points are timed by name, and a refused one is not."""
    import fluxb200 as F
    from fluxb200 import lib
    g = torch.Generator(device="cuda").manual_seed(0)
    x = F.B200Array(torch.randn(64, device="cuda"), (64, 1))
    small, long = _chain(F, [64, 32, 8], "relu", g), _chain(F, [64] * 10, "relu", g)
    prof = {"names": {"fb_dense_chain_fwd", "fb_dense_fwd"}, "events": []}
    monkeypatch.setattr(lib, "PROFILE", prof)
    small(x)
    assert [e[0] for e in prof["events"]] == ["fb_dense_chain_fwd"]
    long(x)
    torch.cuda.synchronize()
    assert [e[0] for e in prof["events"]] == ["fb_dense_chain_fwd"] + ["fb_dense_fwd"] * 9
    assert all(e[2].elapsed_time(e[3]) >= 0 for e in prof["events"])
