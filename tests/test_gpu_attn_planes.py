"""Tensor-core attention (half-precision planes, bf16 planes): head sizes, ragged tiles, unseen keys and slot / region reuse against float64."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# (head size of q / k, of v, heads, Lq, Lk, batch, causal)
CASES = [
    (64, 64, 2, 128, 64, 2, 0), (64, 64, 1, 129, 65, 1, 1), (64, 64, 3, 1, 9, 2, 0), (64, 64, 1, 63, 300, 2, 0), (64, 64, 1, 700, 65, 1, 0),
    (32, 32, 2, 200, 200, 2, 1), (20, 12, 2, 77, 130, 1, 0), (7, 5, 3, 70, 131, 2, 1), (1, 64, 1, 64, 64, 1, 0), (64, 16, 2, 127, 191, 1, 1),
    (64, 64, 1, 100, 400, 1, 1),                                   # keys that no query sees
    (64, 64, 1, 2048, 2112, 1, 0), (64, 64, 1, 2113, 2048, 1, 0),  # the longest accumulations, and one block more
]


def _reference(q, k, v, do, d, dv, heads, causal):
    """out, dq, dk, dv in float64; arrays are [batch][len][heads * size]."""
    q, k, v = (t.double().requires_grad_(True) for t in (q, k, v))
    B, Lq, Lk = q.shape[0], q.shape[1], k.shape[1]
    qh, kh, vh = q.view(B, Lq, heads, d).transpose(1, 2), k.view(B, Lk, heads, d).transpose(1, 2), v.view(B, Lk, heads, dv).transpose(1, 2)
    s = qh @ kh.transpose(2, 3) / np.sqrt(d)
    if causal:
        s = s.masked_fill(torch.arange(Lk, device=s.device)[None, :] > torch.arange(Lq, device=s.device)[:, None], -np.inf)
    out = (torch.softmax(s, -1) @ vh).transpose(1, 2).reshape(B, Lq, heads * dv)
    out.backward(do.double())
    return [t.detach() for t in (out, q.grad, k.grad, v.grad)]


def _err(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


@pytest.mark.parametrize("d,dv,heads,lq,lk,batch,causal", CASES)
@pytest.mark.parametrize("shift", [0, 1])
def test_attention_planes(d, dv, heads, lq, lk, batch, causal, shift):
    """shift = 1: arrays that start 4 bytes past a 16-byte boundary."""
    import fluxb200 as F
    from fluxb200 import lib
    g = torch.Generator(device="cuda")
    g.manual_seed(lq * 7 + lk + d)

    def arr(length, size, fill=True):
        flat = torch.empty(batch * length * size + 4, device="cuda")
        t = flat[shift:shift + batch * length * size].view(batch, length, size)
        return t.normal_(generator=g) if fill else t.fill_(float("nan"))

    q, k, v, do = arr(lq, heads * d), arr(lk, heads * d), arr(lk, heads * dv), arr(lq, heads * dv)
    o, dq, dk, dvv = arr(lq, heads * dv, False), arr(lq, heads * d, False), arr(lk, heads * d, False), arr(lk, heads * dv, False)
    lse = torch.empty(batch * heads * lq, device="cuda")
    ctx = F.context()
    p = [t.data_ptr() for t in (q, k, v)]
    dims = (heads * d, heads * dv, lq, lk, batch, heads, causal)
    lib.call("fb_attn_fwd", ctx.handle, ctx.stream, *p, None, o.data_ptr(), lse.data_ptr(), *dims)
    lib.call("fb_attn_bwd", ctx.handle, ctx.stream, *p, None, o.data_ptr(), lse.data_ptr(), do.data_ptr(), dq.data_ptr(), dk.data_ptr(),
             dvv.data_ptr(), *dims)
    assert ctx.device_error() == 0
    # at most 6 products x 4 steps x 32 blocks truncating adds of 2^-24 into an accumulator, and the scores' own 24: 5e-5
    for name, got, ref in zip(("o", "dq", "dk", "dv"), (o, dq, dk, dvv), _reference(q, k, v, do, d, dv, heads, causal)):
        assert _err(got, ref) < 5e-5, (name, _err(got, ref))


@pytest.mark.parametrize("d,heads,lq,lk,causal", [(64, 2, 129, 65, 1), (64, 1, 1, 9, 0), (32, 3, 300, 300, 1), (8, 2, 700, 131, 0),
                                                  (64, 1, 100, 400, 1), (64, 1, 2048, 2048, 0), (64, 1, 2049, 70, 0)])
def test_attention_bf16(d, heads, lq, lk, causal):
    """bf16 operands through the public call (2049 queries: the backward pass takes the Float32 kernels).  Every output is
    rounded to bf16 once (2^-9 of each value at most): 3e-3 with room for the Float32 sums and the scaled rounding of dO."""
    import fluxb200 as F
    g = torch.Generator(device="cuda")
    g.manual_seed(lq + lk + d)
    batch, E = 2, heads * d
    q, k, v = (torch.randn(batch, n, E, device="cuda", generator=g).bfloat16() for n in (lq, lk, lk))
    arrays = tuple(F.B200Array(t.flatten(), (E, t.shape[1], batch)) for t in (q, k, v))
    mask = F.make_causal_mask() if causal else None

    def f(a):
        y, _ = F.dot_product_attention(*a, nheads=heads, mask=mask)
        return F.sum_abs2(y), y

    (_, y), (grads,) = F.withgradient(f, arrays)
    assert y.t.dtype == torch.bfloat16 and grads[0].t.dtype == torch.bfloat16
    yt = y.t.view(batch, lq, E)
    out, dq, dk, dv = _reference(q, k, v, 2 * yt.double(), d, d, heads, causal)
    for name, got, ref in (("y", yt, out), ("dq", grads[0].t, dq), ("dk", grads[1].t, dk), ("dv", grads[2].t, dv)):
        assert _err(got.view(ref.shape), ref) < 3e-3, (name, _err(got.view(ref.shape), ref))
    plain, alpha = F.dot_product_attention(*arrays, nheads=heads, mask=mask)
    assert torch.equal(plain.t, y.t)
    a = alpha.materialize().t.view(batch, heads, lq, lk)
    assert float((a.sum(-1) - 1).abs().max()) < 1e-4


@pytest.mark.parametrize("d", [8, 16, 24, 32, 40, 48, 56, 64])
@pytest.mark.parametrize("causal", [0, 1])
def test_every_plane_product_is_there(d, causal):
    """Every number of 16-feature steps, one to four key blocks.  The smallest plane products lie near 2^-16 of the whole: one
    that were missing or taken from the wrong place would show as 5e-6 and more.  Forward: 2^-24 for the cut and a few
    roundings to nearest, 5e-7.  Backward at head size 64: 24 truncating adds of 2^-24 a block, 3e-6 for two blocks."""
    import fluxb200 as F
    from fluxb200 import lib
    g = torch.Generator(device="cuda")
    g.manual_seed(d)
    heads, batch = 3, 2
    ctx = F.context()
    for lq, lk in ((128, 64), (200, 120), (64, 250)):
        q, k, v, do = (torch.randn(batch, n, heads * d, device="cuda", generator=g) for n in (lq, lk, lk, lq))
        o, dq, dk, dv = (torch.empty_like(t) for t in (q, q, k, v))
        lse = torch.empty(batch * heads * lq, device="cuda")
        dims = (heads * d, heads * d, lq, lk, batch, heads, causal)
        p = [t.data_ptr() for t in (q, k, v)]
        lib.call("fb_attn_fwd", ctx.handle, ctx.stream, *p, None, o.data_ptr(), lse.data_ptr(), *dims)
        ref = _reference(q, k, v, do, d, d, heads, causal)
        assert _err(o, ref[0]) < 5e-7, _err(o, ref[0])
        if d == 64 and lk <= 128 and lq <= 128:
            lib.call("fb_attn_bwd", ctx.handle, ctx.stream, *p, None, o.data_ptr(), lse.data_ptr(), do.data_ptr(), dq.data_ptr(), dk.data_ptr(),
                     dv.data_ptr(), *dims)
            for name, got, want in zip(("dq", "dk", "dv"), (dq, dk, dv), ref[1:]):
                assert _err(got, want) < 3e-6, (name, _err(got, want))


@pytest.mark.parametrize("lq,lk,causal", [(512, 512, 1), (130, 700, 0)])
def test_backward_of_unaligned_arrays_keeps_float32_sums(lq, lk, causal):
    """Arrays 4 bytes past a 16-byte boundary are the FMA kernels' in the backward pass: two chained sums of at most 700 terms
    with rounding to nearest, sqrt(700) * 2^-24 each = 1.6e-6 of the norm (the plane kernels' truncated sums: 5e-6)."""
    import fluxb200 as F
    from fluxb200 import lib
    g = torch.Generator(device="cuda")
    g.manual_seed(lq)
    heads, d, batch = 4, 64, 2
    mk = lambda n: torch.randn(batch * n * heads * d + 4, device="cuda", generator=g)[1:1 + batch * n * heads * d].view(batch, n, heads * d)
    q, k, v, do, o, dq, dk, dv = (mk(n) for n in (lq, lk, lk, lq, lq, lq, lk, lk))
    lse = torch.empty(batch * heads * lq, device="cuda")
    ctx = F.context()
    dims = (heads * d, heads * d, lq, lk, batch, heads, causal)
    p = [t.data_ptr() for t in (q, k, v)]
    lib.call("fb_attn_fwd", ctx.handle, ctx.stream, *p, None, o.data_ptr(), lse.data_ptr(), *dims)
    lib.call("fb_attn_bwd", ctx.handle, ctx.stream, *p, None, o.data_ptr(), lse.data_ptr(), do.data_ptr(), dq.data_ptr(), dk.data_ptr(),
             dv.data_ptr(), *dims)
    for name, got, ref in zip(("dq", "dk", "dv"), (dq, dk, dv), _reference(q, k, v, do, d, d, heads, causal)[1:]):
        assert _err(got, ref) < 1.6e-6, (name, _err(got, ref))


@pytest.mark.parametrize("d,lq,lk,causal", [(32, 300, 300, 1), (8, 70, 131, 0), (56, 65, 200, 0)])
def test_bf16_backward_of_small_heads_is_the_float32_one(d, lq, lk, causal):
    """Head sizes below 64: the gradients are those of the Float32 kernels on the widened operands, rounded once."""
    import fluxb200 as F
    from fluxb200 import lib
    g = torch.Generator(device="cuda")
    g.manual_seed(d)
    heads, batch = 2, 2
    E = heads * d
    low = tuple(F.B200Array(torch.randn(batch * n * E, device="cuda", generator=g).bfloat16(), (E, n, batch)) for n in (lq, lk, lk))
    mask = F.make_causal_mask() if causal else None
    ctx = F.context()
    dims = (E, E, lq, lk, batch, heads, causal)
    (_, y), (grads,) = F.withgradient(lambda a: (lambda y: (F.sum_abs2(y), y))(F.dot_product_attention(*a, nheads=heads, mask=mask)[0]), low)
    q, k, v = (t.t.float() for t in low)
    o32, o16 = torch.empty(batch * lq * E, device="cuda"), torch.empty(batch * lq * E, device="cuda", dtype=torch.bfloat16)
    lse = torch.empty(batch * heads * lq, device="cuda")
    lib.call("fb_attn_fwd_bf16", ctx.handle, ctx.stream, *[t.ptr for t in low], o32.data_ptr(), o16.data_ptr(), lse.data_ptr(), *dims)
    assert torch.equal(o16, y.t)
    do = (2 * y.t.float()).bfloat16().float()
    out = [torch.empty_like(t) for t in (q, k, v)]
    lib.call("fb_attn_bwd", ctx.handle, ctx.stream, *[t.data_ptr() for t in (q, k, v)], None, o32.data_ptr(), lse.data_ptr(), do.data_ptr(),
             *[t.data_ptr() for t in out], *dims)
    for got, ref in zip(grads, out):
        assert torch.equal(got.t, ref.bfloat16())


@pytest.mark.parametrize("d,dv,lq,lk,causal,shift,dtype", [(32, 32, 200, 300, 0, 0, "f32"), (20, 12, 77, 130, 1, 0, "f32"), (64, 64, 300, 129, 0, 1, "f32"),
                                                           (64, 16, 65, 64, 1, 0, "f32"), (32, 32, 200, 300, 0, 0, "bf16"), (8, 16, 129, 70, 1, 0, "bf16")])
def test_infinite_and_nan_operands(d, dv, lq, lk, causal, shift, dtype):
    """What the FMA kernel (reached through an additive bias of zeros) makes of operands that are not finite, bit for bit, in
    the heads that hold them; the other heads are as they are without them."""
    import fluxb200 as F
    from fluxb200 import lib
    g = torch.Generator(device="cuda")
    g.manual_seed(d + lq)
    heads, batch, inf = 4, 2, float("inf")
    mk = lambda n, size: torch.randn(batch * n * heads * size + 4, device="cuda", generator=g)[shift:shift + batch * n * heads * size].view(batch, n, heads, size)
    clean = [mk(lq, d), mk(lk, d), mk(lk, dv)]
    if dtype == "bf16":
        clean = [t.bfloat16().float() for t in clean]
    ctx = F.context()
    dims = (heads * d, heads * dv, lq, lk, batch, heads, causal)
    zero_bias = torch.zeros(lk * lq, device="cuda")

    def forward(arrays, general=False):
        o, lse = mk(lq, dv), torch.empty(batch, heads, lq, device="cuda")
        if dtype == "bf16" and not general:
            low, o16 = [t.bfloat16() for t in arrays], torch.empty(o.shape, device="cuda", dtype=torch.bfloat16)
            lib.call("fb_attn_fwd_bf16", ctx.handle, ctx.stream, *[t.data_ptr() for t in low], o.data_ptr(), o16.data_ptr(), lse.data_ptr(), *dims)
            assert torch.equal(torch.nan_to_num(o16), torch.nan_to_num(o.bfloat16()))
            return o, lse
        lib.call("fb_attn_fwd_ex", ctx.handle, ctx.stream, *[t.data_ptr() for t in arrays], None, zero_bias.data_ptr() if general else None, 0, 0,
                 0.0, 0, 0, o.data_ptr(), lse.data_ptr(), *dims)
        return o, lse
    plain, plain_lse = forward(clean)
    arrays = [t.clone() if not shift else mk(t.shape[1], t.shape[3]).copy_(t) for t in clean]
    arrays[0][0, lq // 2, 0, 1] = inf                # a query
    arrays[1][0, lk // 3, 1, 0] = -inf               # a key: weight 0 or 1, by the sign of the query's value
    arrays[2][1, 3, 2, dv - 1] = inf                 # a value
    arrays[1][1, lk - 1, 3, d - 1] = float("nan")
    (o, lse), (ref, ref_lse) = forward(arrays), forward(arrays, general=True)
    touched = {(0, 0), (0, 1), (1, 2), (1, 3)}
    for b in range(batch):
        for h in range(heads):
            if (b, h) in touched:
                assert torch.equal(torch.isnan(o[b, :, h]), torch.isnan(ref[b, :, h]))
                assert torch.equal(torch.nan_to_num(o[b, :, h], nan=7.0), torch.nan_to_num(ref[b, :, h], nan=7.0))
                assert torch.equal(torch.nan_to_num(lse[b, h], nan=7.0), torch.nan_to_num(ref_lse[b, h], nan=7.0))
            else:
                assert torch.equal(o[b, :, h], plain[b, :, h]) and torch.equal(lse[b, h], plain_lse[b, h])
    assert bool(torch.isinf(ref[1, 3:, 2, dv - 1]).any()) and bool(torch.isfinite(ref[0, :, 1]).any())
    assert ctx.device_error() == 0


def test_attention_two_streams():
    """Calls of one thread on two streams take their operand images from one pool: neither may read the other's."""
    import fluxb200 as F
    from fluxb200 import lib
    heads, d, n, batch = 8, 64, 512, 4
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    dims = (heads * d, heads * d, n, n, batch, heads, 0)
    ctx = F.context()
    sets = []
    for _ in range(2):
        q, k, v = (torch.randn(batch, n, heads * d, device="cuda", generator=g) for _ in range(3))
        sets.append((q, k, v, torch.empty_like(q), torch.empty(batch * heads * n, device="cuda"), torch.empty_like(q)))

    def forward(s, out, stream):
        lib.call("fb_attn_fwd", ctx.handle, stream, *[t.data_ptr() for t in s[:3]], None, out.data_ptr(), s[4].data_ptr(), *dims)

    for s in sets:
        forward(s, s[5], ctx.stream)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(20):
        for s, st in zip(sets, streams):
            forward(s, s[3], st.cuda_stream)
    torch.cuda.synchronize()
    for s in sets:
        assert torch.equal(s[3], s[5])


def _forward_set(g, batch, n, heads, d):
    q, k, v = (torch.randn(batch, n, heads * d, device="cuda", generator=g) for _ in range(3))
    return q, k, v, torch.empty_like(q), torch.empty(batch * heads * n, device="cuda"), torch.empty_like(q)


def test_attention_replay_beside_eager_calls():
    """A replayed graph and eager calls (or another replay) on two streams: a captured call's images are its graph's own."""
    import fluxb200 as F
    from fluxb200 import lib
    heads, d, n, batch = 8, 64, 512, 4
    g = torch.Generator(device="cuda")
    g.manual_seed(6)
    dims = (heads * d, heads * d, n, n, batch, heads, 0)
    ctx = F.context()
    sets = [_forward_set(g, batch, n, heads, d) for _ in range(3)]

    def forward(s, out):
        lib.call("fb_attn_fwd", ctx.handle, ctx.stream, *[t.data_ptr() for t in s[:3]], None, out.data_ptr(), s[4].data_ptr(), *dims)
    for s in sets:
        forward(s, s[5])
    torch.cuda.synchronize()
    graphs = []
    for s in sets[:2]:
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            for _ in range(3):
                forward(s, s[3])
    streams = [torch.cuda.Stream() for _ in range(3)]
    for _ in range(10):
        for graph, st in zip(graphs, streams):
            with torch.cuda.stream(st):
                graph.replay()
        with torch.cuda.stream(streams[2]):
            for _ in range(3):
                forward(sets[2], sets[2][3])
    torch.cuda.synchronize()
    for s in sets:
        assert torch.equal(s[3], s[5])


def test_attention_captured_without_warm_up():
    """A context whose first attention call of a size is inside a capture runs the same kernels there as eagerly."""
    import fluxb200 as F
    from fluxb200 import core, lib
    heads, d, n, batch = 4, 64, 700, 3
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    dims = (heads * d, heads * d, n, n, batch, heads, 1)
    ctx, fresh = F.context(), core.Context(0)
    q, k, v, o, lse, ref = _forward_set(g, batch, n, heads, d)
    do = torch.randn(q.shape, device="cuda", generator=g)
    grads, ref_grads = [[torch.empty_like(q) for _ in range(3)] for _ in range(2)]

    def both(handle, out, gr):
        p = [t.data_ptr() for t in (q, k, v)]
        lib.call("fb_attn_fwd", handle, ctx.stream, *p, None, out.data_ptr(), lse.data_ptr(), *dims)
        lib.call("fb_attn_bwd", handle, ctx.stream, *p, None, out.data_ptr(), lse.data_ptr(), do.data_ptr(), *[t.data_ptr() for t in gr], *dims)
    both(ctx.handle, ref, ref_grads)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        both(fresh.handle, o, grads)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(o, ref) and all(torch.equal(a, b) for a, b in zip(grads, ref_grads))
    del graph
    lib.call("fb_ctx_destroy", fresh.handle)


def _skewed(kind, q, k, v, do, heads):
    """Inputs of which half-precision planes would lose something: heads that hold such values are computed on three bf16 planes."""
    if kind == "graded":           # every third feature 2^30 larger in K and V, and as much smaller in Q and dO
        s = torch.ones(q.shape[-1], device=q.device)
        s[::3] = 2.0 ** 30
        return q / s, k * s, v * s, do / s
    if kind == "one head":         # the same in the last head alone
        s = torch.ones(q.shape[-1], device=q.device)
        s[-q.shape[-1] // heads::3] = 2.0 ** 36
        return q / s, k * s, v * s, do / s
    if kind == "late gradient":    # tiles of dO whose scales lie far apart
        return q, k, v, do * torch.exp2(-torch.arange(do.shape[1], device=q.device) / 4.0)[None, :, None]
    if kind == "one query":        # tiles of zeros
        do = do.clone()
        do[:, :-1] = 0
        return q, k, v, do
    if kind == "large":            # shifts beyond their limits
        return q * 2.0 ** -70, k * 2.0 ** 70, v * 2.0 ** 50, do
    return q, k, v, do * 2.0 ** -80


@pytest.mark.parametrize("kind", ["graded", "one head", "late gradient", "one query", "large", "small gradient"])
@pytest.mark.parametrize("heads,lq,lk,batch,causal", [(2, 300, 300, 2, 1), (3, 130, 450, 1, 0), (1, 64, 64, 1, 0)])
@pytest.mark.parametrize("low", [False, True])
def test_inputs_of_very_different_magnitudes(kind, heads, lq, lk, batch, causal, low):
    """Feature by feature: gradients of the graded inputs are as exact as those of ordinary ones.  Bounds: 5e-5 as above; bf16 results
    are rounded to 2^-9."""
    import fluxb200 as F
    from fluxb200 import lib
    g, E, ctx = torch.Generator(device="cuda").manual_seed(lq), 64 * heads, F.context()
    q, k, v, do = (torch.randn(batch, n, E, generator=g, device="cuda") for n in (lq, lk, lk, lq))
    q, k, v, do = (t.contiguous() for t in _skewed(kind, q, k, v, do, heads))
    dims, lse, o = (E, E, lq, lk, batch, heads, causal), torch.empty(batch * heads * lq, device="cuda"), torch.empty_like(q)
    p = lambda t: t.data_ptr()
    if low:
        q, k, v, do = (t.bfloat16() for t in (q, k, v, do))
        out, dq, dk, dv = (torch.empty_like(t) for t in (q, q, k, v))
        lib.call("fb_attn_fwd_bf16", ctx.handle, ctx.stream, p(q), p(k), p(v), p(o), p(out), p(lse), *dims)
        lib.call("fb_attn_bwd_bf16", ctx.handle, ctx.stream, p(q), p(k), p(v), p(o), p(lse), p(do), p(dq), p(dk), p(dv), *dims)
    else:
        dq, dk, dv = (torch.empty_like(t) for t in (q, k, v))
        lib.call("fb_attn_fwd", ctx.handle, ctx.stream, p(q), p(k), p(v), None, p(o), p(lse), *dims)
        lib.call("fb_attn_bwd", ctx.handle, ctx.stream, p(q), p(k), p(v), None, p(o), p(lse), p(do), p(dq), p(dk), p(dv), *dims)
    assert ctx.device_error() == 0
    ref = _reference(q, k, v, do, 64, 64, heads, causal)
    for name, got, want in zip(("o", "dq", "dk", "dv"), (o, dq, dk, dv), ref):
        tol = 1e-2 if low and name != "o" else 5e-5
        got, want = got.double().reshape(-1, E), want.reshape(-1, E)
        if kind == "one query":    # (a feature of dQ is then one element, a sum that may cancel)
            got, want = got.reshape(-1, 1), want.reshape(-1, 1)
        err = float(((got - want).norm(dim=0) / want.norm(dim=0).clamp_min(1e-300)).max())
        assert err < tol, (name, err)


@pytest.mark.parametrize("scores", [16, 24])
@pytest.mark.parametrize("heads,n,batch,causal", [(2, 512, 1, 1), (3, 1000, 2, 1)])
def test_bf16_gradients_of_values_with_small_weights(scores, heads, n, batch, causal):
    """Scores of standard deviation 16 and 24: keys whose largest weight is as small as 2^-80.  Their own rows of dV are as exact as the
    others': the one rounding to bf16 (2^-9) and as much again for scores of up to 130 and truncated sums."""
    import fluxb200 as F
    from fluxb200 import lib
    g, E, ctx = torch.Generator(device="cuda").manual_seed(n), 64 * heads, F.context()
    q, k, v, do = ((torch.randn(batch, n, E, generator=g, device="cuda") * s).bfloat16() for s in (scores ** 0.5, scores ** 0.5, 1.0, 1.0))
    o, lse, out, dq, dk, dv = torch.empty(batch, n, E, device="cuda"), torch.empty(batch * heads * n, device="cuda"), *(torch.empty_like(q) for _ in range(4))
    p, dims = lambda t: t.data_ptr(), (E, E, n, n, batch, heads, causal)
    lib.call("fb_attn_fwd_bf16", ctx.handle, ctx.stream, p(q), p(k), p(v), p(o), p(out), p(lse), *dims)
    lib.call("fb_attn_bwd_bf16", ctx.handle, ctx.stream, p(q), p(k), p(v), p(o), p(lse), p(do), p(dq), p(dk), p(dv), *dims)
    assert ctx.device_error() == 0
    ref = _reference(q, k, v, do, 64, 64, heads, causal)
    split = lambda t: t.double().view(batch, n, heads, 64).transpose(1, 2)
    s = split(q) @ split(k).transpose(2, 3) / 8
    if causal:
        s = s.masked_fill(torch.arange(n, device="cuda")[None, :] > torch.arange(n, device="cuda")[:, None], -np.inf)
    counts = torch.softmax(s, -1).amax(2) > 2.0 ** -80     # [batch][head][key]
    assert bool((torch.softmax(s, -1).amax(2)[counts] < 2.0 ** -50).any())
    got, want = split(dv)[counts], split(ref[3])[counts]
    err = float(((got - want).norm(dim=1) / want.norm(dim=1)).max())
    assert err < 4e-3, err


def _f32_call(q, k, v, do, d, dv, heads, causal):
    """[o, lse, dq, dk, dv] through the Float32 entry points."""
    import fluxb200 as F
    from fluxb200 import lib
    ctx, (batch, lq, _), lk = F.context(), q.shape, k.shape[1]
    p, dims = lambda t: t.data_ptr(), (heads * d, heads * dv, lq, lk, batch, heads, causal)
    o, lse = torch.full_like(do, float("nan")), torch.full((batch * heads * lq,), float("nan"), device="cuda")
    dq, dk, dvv = (torch.full_like(t, float("nan")) for t in (q, k, v))
    lib.call("fb_attn_fwd", ctx.handle, ctx.stream, p(q), p(k), p(v), None, p(o), p(lse), *dims)
    lib.call("fb_attn_bwd", ctx.handle, ctx.stream, p(q), p(k), p(v), None, p(o), p(lse), p(do), p(dq), p(dk), p(dvv), *dims)
    assert ctx.device_error() == 0
    return [o, lse, dq, dk, dvv]


@pytest.mark.parametrize("d,dv,heads,lq,lk,batch,causal", CASES)
@pytest.mark.parametrize("shift", [0, 1])
def test_heads_with_large_scores(d, dv, heads, lq, lk, batch, causal, shift):
    """Scores eight times the ordinary ones: heads of three bf16 planes.  5e-5 as for the ordinary ones."""
    g = torch.Generator(device="cuda").manual_seed(lq + 3 * lk + d)
    mk = lambda n, size, s=1.0: (torch.randn(batch * n * size + 4, device="cuda", generator=g) * s)[shift:shift + batch * n * size].view(batch, n, size)
    q, k, v, do = mk(lq, heads * d, 8.0), mk(lk, heads * d), mk(lk, heads * dv), mk(lq, heads * dv)
    o, _, dq, dk, dvv = _f32_call(q, k, v, do, d, dv, heads, causal)
    for name, got, ref in zip(("o", "dq", "dk", "dv"), (o, dq, dk, dvv), _reference(q, k, v, do, d, dv, heads, causal)):
        assert _err(got, ref) < 5e-5, (name, _err(got, ref))


@pytest.mark.parametrize("heads,n,batch", [(2, 512, 1), (3, 300, 2)])
def test_a_key_and_a_value_far_above_the_others(heads, n, batch):
    """One key 1e4 times the others (and read by a feature of Q as much smaller), one value 1e4 times: scores of some thousand, in which 2^-24
    of the operands is 1e-4 of a weight.  Three bf16 planes: output 6e-7, dQ 1.6e-4, dV 2.5e-4 (23 bits: 3.6e-6, 4.3e-3, 1.7e-3)."""
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v, do = (torch.randn(batch, n, 64 * heads, device="cuda", generator=g) for _ in range(4))
    k[:, 5] *= 1e4
    q[:, :, ::64] *= 1e-4
    v[:, 7] *= 1e4
    o, _, dq, dk, dv = _f32_call(q, k, v, do, 64, 64, heads, 1)
    ref = _reference(q, k, v, do, 64, 64, heads, 1)
    for name, got, want, tol in zip(("o", "dq", "dk", "dv"), (o, dq, dk, dv), ref, (1.5e-6, 5e-4, 2e-5, 7e-4)):
        assert _err(got, want) < tol, (name, _err(got, want))


@pytest.mark.parametrize("heads,lq,lk,batch,causal", [(2, 300, 300, 2, 1), (3, 130, 450, 1, 0), (1, 64, 64, 1, 0), (2, 1, 9, 3, 0), (1, 700, 65, 1, 1), (2, 2048, 2048, 1, 1)])
def test_picked_heads_have_the_bits_of_bf16_operands(heads, lq, lk, batch, causal):
    """Float32 operands that are bf16 values: their lower planes are zeros, which add nothing, so outputs and gradients are those of the bf16
    entry points before their rounding."""
    import fluxb200 as F
    from fluxb200 import lib
    g = torch.Generator(device="cuda").manual_seed(lq)
    E, ctx = 64 * heads, F.context()
    low = [(torch.randn(batch, n, E, device="cuda", generator=g) * s).bfloat16() for n, s in ((lq, 9.0), (lk, 1.0), (lk, 1.0), (lq, 1.0))]
    o, lse, dq, dk, dv = _f32_call(*[t.float() for t in low], 64, 64, heads, causal)
    q, k, v, do = low
    p, dims = lambda t: t.data_ptr(), (E, E, lq, lk, batch, heads, causal)
    o32, l32, out, rq, rk, rv = torch.empty_like(o), torch.empty_like(lse), *(torch.empty_like(t) for t in (q, q, k, v))
    lib.call("fb_attn_fwd_bf16", ctx.handle, ctx.stream, p(q), p(k), p(v), p(o32), p(out), p(l32), *dims)
    lib.call("fb_attn_bwd_bf16", ctx.handle, ctx.stream, p(q), p(k), p(v), p(o32), p(l32), p(do), p(rq), p(rk), p(rv), *dims)
    assert torch.equal(o, o32) and torch.equal(lse, l32) and torch.equal(o.bfloat16(), out)
    for got, want in ((dq, rq), (dk, rk), (dv, rv)):
        assert torch.equal(got.bfloat16(), want)


@pytest.mark.parametrize("heads,n,batch,causal,shift", [(16, 2048, 4, 1, 0), (5, 200, 3, 0, 0), (7, 130, 2, 1, 1), (33, 64, 40, 0, 0), (16, 1024, 45, 0, 0)])
@pytest.mark.parametrize("which", ["all", "some", "none of the first"])
def test_heads_are_picked_one_by_one(heads, n, batch, causal, shift, which):
    """A head has the bits that it has in a call of its own, whatever the others are: up to eight picked tiles a CTA, none, and a few; images of
    three chunks of the batch (the last size)."""
    g = torch.Generator(device="cuda").manual_seed(heads)
    mk = lambda: torch.randn(batch * n * heads * 64 + 4, device="cuda", generator=g)[shift:shift + batch * n * heads * 64].view(batch, n, heads, 64)
    q, k, v, do = mk(), mk(), mk(), mk()
    large = torch.zeros(batch, heads, dtype=torch.bool, device="cuda")
    if which == "all":
        large[:] = True
    elif which == "some":
        large.view(-1)[::7] = True
        large.view(-1)[3] = True
    else:
        large.view(-1)[-1] = True
    q[:] = torch.where(large[:, None, :, None], q * 12.0, q)
    flat = lambda t: t.reshape(batch, n, heads * 64) if not shift else t.view(batch, n, heads * 64)
    got = _f32_call(*map(flat, (q, k, v, do)), 64, 64, heads, causal)
    lse = got[1].view(batch, heads, n)
    for b, h in ((0, 0), (0, 3), (batch - 1, heads - 1), (batch // 2, heads // 2)):
        alone = _f32_call(*(t[b:b + 1, :, h].contiguous() for t in (q, k, v, do)), 64, 64, 1, causal)
        assert torch.equal(lse[b, h], alone[1])
        if shift:      # (unaligned arrays have the FMA kernels' gradients)
            alone = alone[:1]
        for a, r in zip([got[0]] + got[2:], [alone[0]] + alone[2:]):
            assert torch.equal(a.view(batch, n, heads, 64)[b, :, h], r[0])


@pytest.mark.parametrize("what,picked", [("one faint element", False), ("a faint row", True), ("a faint column", True), ("a row of zeros", False), ("tails", False)])
@pytest.mark.parametrize("operand", [0, 1, 2, 3])
def test_which_tiles_the_planes_hold(what, picked, operand):
    """A position or a feature far below the rest of its tile makes its head one of three bf16 planes; single small elements and zeros do not.
    Row by row and column by column the results are as exact as ordinary ones (5e-5; forward 2e-6)."""
    g = torch.Generator(device="cuda").manual_seed(operand)
    n, heads = 192, 2
    x = [torch.randn(1, n, 64 * heads, device="cuda", generator=g) for _ in range(4)]
    t = x[operand]
    if what == "one faint element":
        t[0, 70, 3] = 1e-9
    elif what == "a faint row":
        t[0, 70, :64] *= 2.0 ** -24
    elif what == "a faint column":
        t[0, 64:128, 3] *= 2.0 ** -24
    elif what == "a row of zeros":
        t[0, 70] = 0.0
    else:
        t[:] = torch.nn.functional.gelu(3.0 * t)
    got = _f32_call(*x, 64, 64, heads, 0)
    ref = _reference(*x, 64, 64, heads, 0)
    for i, (name, a, r) in enumerate(zip(("o", "dq", "dk", "dv"), [got[0]] + got[2:], ref)):
        a, r = a.double().view(n, heads, 64), r.view(n, heads, 64)
        for dim in (0, 2):
            keep = r.abs().amax(dim) > 0
            err = ((a - r).norm(dim=dim) / r.norm(dim=dim).clamp_min(1e-300))[keep].max()
            assert float(err) < (2e-6 if i == 0 else 5e-5), (name, dim, float(err))
    # (three planes hold every exponent: powers of two moved from K to Q change no bit of a picked head)
    if not picked:
        return
    s = 2.0 ** 9
    same = _f32_call(x[0] * s, x[1] / s, x[2], x[3], 64, 64, heads, 0)
    assert torch.equal(same[0].view(n, heads, 64)[:, 0], got[0].view(n, heads, 64)[:, 0])


def test_a_replayed_graph_picks_anew():
    """Which heads are picked is decided on the device: a graph captured with ordinary inputs gives what an eager call gives of others."""
    import fluxb200 as F
    from fluxb200 import lib
    g = torch.Generator(device="cuda").manual_seed(2)
    heads, n, batch = 4, 300, 2
    sets = [[torch.randn(batch, n, heads * 64, device="cuda", generator=g) for _ in range(4)] for _ in range(3)]
    sets[1][0][0, :, :64] *= 12.0
    sets[2][0] *= 12.0
    want = [_f32_call(*s, 64, 64, heads, 1) for s in sets]
    q, k, v, do = (t.clone() for t in sets[0])
    o, lse = torch.empty_like(q), torch.empty(batch * heads * n, device="cuda")
    dq, dk, dv = (torch.empty_like(t) for t in (q, k, v))
    ctx, p, dims = F.context(), lambda t: t.data_ptr(), (heads * 64, heads * 64, n, n, batch, heads, 1)

    def call():
        lib.call("fb_attn_fwd", ctx.handle, ctx.stream, p(q), p(k), p(v), None, p(o), p(lse), *dims)
        lib.call("fb_attn_bwd", ctx.handle, ctx.stream, p(q), p(k), p(v), None, p(o), p(lse), p(do), p(dq), p(dk), p(dv), *dims)
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for s, ref in list(zip(sets, want)) * 2:
        for t, new in zip((q, k, v, do), s):
            t.copy_(new)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip((o, lse, dq, dk, dv), ref))
    assert ctx.device_error() == 0


@pytest.mark.parametrize("lq,lk,causal,low", [(200, 300, 0, False), (130, 130, 1, False), (200, 300, 0, True), (130, 130, 1, True), (2100, 70, 0, False), (70, 2100, 0, False)])
def test_gradients_of_heads_that_are_not_finite(lq, lk, causal, low):
    """Heads with an infinite or NaN operand have the gradients of the FMA kernels (reached through an additive bias of zeros): the same values
    are finite, and those agree as Float32 sums in two orders do (2e-5 of the head; bf16 results 2^-8).  The other heads keep their bits."""
    import fluxb200 as F
    from fluxb200 import lib
    g = torch.Generator(device="cuda").manual_seed(lq)
    heads, batch, inf = 5, 2, float("inf")
    E, ctx = 64 * heads, F.context()
    p, dims = lambda t: t.data_ptr(), (E, E, lq, lk, batch, heads, causal)
    x = [torch.randn(batch, n, heads, 64, device="cuda", generator=g) for n in (lq, lk, lk, lq)]
    if low:
        x = [t.bfloat16().float() for t in x]
    zero_bias = torch.zeros(lk * lq, device="cuda")

    def gradients(q, k, v, do, general):
        o, lse = torch.empty(batch, lq, E, device="cuda"), torch.empty(batch * heads * lq, device="cuda")
        if low and not general:
            q, k, v, do = (t.bfloat16() for t in (q, k, v, do))
            out, dq, dk, dv = (torch.empty_like(t) for t in (q, q, k, v))
            lib.call("fb_attn_fwd_bf16", ctx.handle, ctx.stream, p(q), p(k), p(v), p(o), p(out), p(lse), *dims)
            lib.call("fb_attn_bwd_bf16", ctx.handle, ctx.stream, p(q), p(k), p(v), p(o), p(lse), p(do), p(dq), p(dk), p(dv), *dims)
        else:
            dq, dk, dv = (torch.empty_like(t) for t in (q, k, v))
            b = p(zero_bias) if general else None
            lib.call("fb_attn_fwd_ex", ctx.handle, ctx.stream, p(q), p(k), p(v), None, b, 0, 0, 0.0, 0, 0, p(o), p(lse), *dims)
            lib.call("fb_attn_bwd_ex", ctx.handle, ctx.stream, p(q), p(k), p(v), None, b, 0, 0, 0.0, 0, 0, p(o), p(lse), p(do), None, p(dq), p(dk), p(dv), *dims)
        assert ctx.device_error() == 0
        return [t.view(batch, -1, heads, 64).float() for t in (dq, dk, dv)]
    clean = gradients(*x, False)
    bad = [t.clone() for t in x]
    bad[0][0, lq // 2, 0, 1] = inf
    bad[1][0, lk // 3, 1, 0] = -inf
    bad[2][1, 3, 2, 5] = inf
    bad[3][1, lq - 1, 3, 7] = float("nan")
    got, ref = gradients(*bad, False), gradients(*bad, True)
    touched = {(0, 0), (0, 1), (1, 2), (1, 3)}
    for name, a, r, c in zip(("dq", "dk", "dv"), got, ref, clean):
        for b in range(batch):
            for h in range(heads):
                if (b, h) not in touched:
                    assert torch.equal(a[b, :, h], c[b, :, h]), (name, b, h)
                    continue
                fine = torch.isfinite(r[b, :, h])
                assert torch.equal(torch.isfinite(a[b, :, h]), fine), (name, b, h)
                if bool(fine.any()):
                    err = float((a[b, :, h] - r[b, :, h])[fine].abs().max() / r[b, :, h][fine].abs().max().clamp_min(1e-30))
                    assert err < (2.0 ** -8 if low else 2e-5), (name, b, h, err)
