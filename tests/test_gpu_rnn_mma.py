"""GPU tests of the tensor-core recurrences at the edges of their cuts: hidden sizes around 16 units, 128 / 256 / 512 (k-steps per warp)
and the backward pieces of 64, batches around 8 and 16 columns and of several chunks per CTA, initial states, steps that
send nothing.  Reference: float64 autograd.

Tolerance: operands rounded to 23 bits and sums of up to 2048 Float32 products, partly truncated, through up to 40 dependent steps
whose gates have slopes below one: 5e-6 of the largest value; 2e-5 on what is summed over steps and batch."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (sequences of T * H >= 1536 and 48 <= H <= 512 take them; the others here are the neighbours across those lines)
SHAPES = [(1, 1, 2), (47, 7, 33), (48, 8, 32), (49, 9, 32), (64, 17, 24), (127, 5, 13), (128, 16, 12), (129, 33, 12), (255, 3, 7), (256, 65, 6),
          (257, 8, 6), (340, 40, 5), (511, 20, 4), (512, 64, 4), (512, 150, 3), (512, 2, 2), (500, 1, 40), (96, 12, 17), (80, 300, 20), (48, 700, 32),
          (200, 20, 8), (513, 9, 3)]


def _reference(cell, wi, wh, b, x, h, c):
    out, gx = [], x @ wi + b
    for t in range(x.shape[1]):
        gh = h @ wh
        if cell == "lstm":
            i, f, g, o = (gx[:, t] + gh).chunk(4, 1)
            c = torch.sigmoid(f) * c + torch.sigmoid(i) * torch.tanh(g)
            h = torch.sigmoid(o) * torch.tanh(c)
        else:
            (a1, a2, a3), (g1, g2, g3) = gx[:, t].chunk(3, 1), gh.chunk(3, 1)
            r, z = torch.sigmoid(a1 + g1), torch.sigmoid(a2 + g2)
            h = (1 - z) * torch.tanh(a3 + r * g3) + z * h
        out.append(h)
    return torch.stack(out, 1), h, c


@pytest.mark.parametrize("cell", ["lstm", "gru"])
@pytest.mark.parametrize("states", [False, True])
@pytest.mark.parametrize("H,B,T", SHAPES)
def test_recurrences(cell, states, H, B, T):
    import fluxb200 as F
    from fluxb200 import lib
    ctx, I, ng = F.context(0), 12, 4 if cell == "lstm" else 3
    g = torch.Generator(device="cuda").manual_seed(H + B + T)
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    p = lambda t: None if t is None else t.data_ptr()
    wi, wh, b = new(I, ng * H) / I ** 0.5, new(H, ng * H) / H ** 0.5, new(ng * H) * 0.1
    wh[:, ::7] *= 2.0 ** -20                          # gate rows of very different magnitude
    x, dout = new(B, T, I), new(B, T, H)
    dout[B // 2] *= 2.0 ** 30                         # and columns
    h0, c0 = (new(B, H) * 3, new(B, H) if cell == "lstm" else None) if states else (None, None)
    dhT, dcT = (new(B, H), new(B, H)) if states else (None, None)
    out, hT, cT = torch.empty(B, T, H, device="cuda"), torch.empty(B, H, device="cuda"), torch.empty(B, H, device="cuda")
    dwi, dwh, db, dx = (torch.empty_like(t) for t in (wi, wh, b, x))
    alone = torch.empty_like(out)
    if cell == "lstm":
        cache = torch.empty(lib.raw().fb_lstm_cache_bytes(I, H, T, B) // 4, device="cuda")
        lib.call("fb_lstm_fwd", ctx.handle, ctx.stream, p(wi), p(wh), p(b), p(x), p(h0), p(c0), p(out), p(hT), p(cT), p(cache), I, H, T, B)
        lib.call("fb_lstm_bwd", ctx.handle, ctx.stream, p(wi), p(wh), p(x), p(h0), p(c0), p(out), p(cache), p(dout), p(dhT), p(dcT), p(dwi), p(dwh),
                 p(db), p(dx), I, H, T, B)
        lib.call("fb_lstm_fwd", ctx.handle, ctx.stream, p(wi), p(wh), p(b), p(x), p(h0), p(c0), p(alone), None, None, None, I, H, T, B)
    else:
        cache = torch.empty(lib.raw().fb_gru_cache_bytes(I, H, T, B) // 4, device="cuda")
        lib.call("fb_gru_fwd", ctx.handle, ctx.stream, p(wi), p(wh), p(b), p(x), p(h0), p(out), p(hT), p(cache), I, H, T, B)
        lib.call("fb_gru_bwd", ctx.handle, ctx.stream, p(wi), p(wh), p(x), p(h0), p(out), p(cache), p(dout), p(dhT), p(dwi), p(dwh), p(db), p(dx), I, H, T, B)
        lib.call("fb_gru_fwd", ctx.handle, ctx.stream, p(wi), p(wh), p(b), p(x), p(h0), p(alone), None, None, I, H, T, B)
    assert ctx.device_error() == 0 and torch.equal(alone, out)
    leaf = lambda t: t.double().requires_grad_()
    rwi, rwh, rb, rx = map(leaf, (wi, wh, b, x))
    zero = torch.zeros(B, H, device="cuda", dtype=torch.double)
    ref, rh, rc = _reference(cell, rwi, rwh, rb, rx, h0.double() if states else zero, c0.double() if c0 is not None else zero)
    total = (ref * dout.double()).sum()
    if states:
        total = total + (rh * dhT.double()).sum() + ((rc * dcT.double()).sum() if cell == "lstm" else 0.0)
    total.backward()

    def close(got, want, tol, name):
        err = float((got.double() - want).abs().max() / want.abs().max())
        assert err < tol, (name, err)
    close(out, ref.detach(), 5e-6, "out")
    close(hT, rh.detach(), 5e-6, "hT")
    if cell == "lstm":
        close(cT, rc.detach(), 5e-6, "cT")
    for got, want, name in ((dwi, rwi, "dWi"), (dwh, rwh, "dWh"), (db, rb, "db")):
        if name != "dWh" or T > 1 or states:
            close(got, want.grad, 2e-5, name)
    for i in range(B):                                # every column by its own largest value
        close(dx[i], rx.grad[i], 2e-5, "dx")


@pytest.mark.parametrize("cell", ["lstm", "gru"])
@pytest.mark.parametrize("H,B,T", [(512, 40, 37), (400, 130, 27), (500, 9, 130), (512, 150, 13)])
def test_backward_slots_that_are_reset(cell, H, B, T):
    """Exchanges of more than 32 MB: twelve slots take the steps in turn (the last shape: one slot is used twice)."""
    test_recurrences(cell, False, H, B, T)


def test_a_sequence_inside_a_graph_beside_another_stream():
    """The exchange buffer belongs to the call: replays and eager calls on another stream give what each gives alone."""
    import fluxb200 as F
    from fluxb200 import lib
    ctx = F.context(0)
    g = torch.Generator(device="cuda").manual_seed(0)
    H, B, T, I = 96, 12, 20, 16
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    wi, wh, b = new(I, 4 * H) / 4, new(H, 4 * H) / 10, new(4 * H) * 0.1
    xs = [new(B, T, I), new(B, T, I)]
    outs = [torch.empty(B, T, H, device="cuda") for _ in range(2)]
    caches = [torch.empty(lib.raw().fb_lstm_cache_bytes(I, H, T, B) // 4, device="cuda") for _ in range(2)]

    def call(k):
        lib.call("fb_lstm_fwd", ctx.handle, ctx.stream, wi.data_ptr(), wh.data_ptr(), b.data_ptr(), xs[k].data_ptr(), None, None, outs[k].data_ptr(), None, None,
                 caches[k].data_ptr(), I, H, T, B)
    want = []
    for k in range(2):
        call(k)
        torch.cuda.synchronize()
        want.append(outs[k].clone())
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph):
        call(0)
    torch.cuda.synchronize()
    for _ in range(5):
        outs[0].zero_()
        outs[1].zero_()
        torch.cuda.synchronize()
        graph.replay()
        with torch.cuda.stream(side):
            call(1)
        torch.cuda.synchronize()
        assert torch.equal(outs[0], want[0]) and torch.equal(outs[1], want[1]) and ctx.device_error() == 0


def _forward(cell, wi, wh, b, x, h0, c0=None):
    import fluxb200 as F
    from fluxb200 import lib
    ctx, (B, T, I), H = F.context(0), x.shape, wh.shape[0]
    p = lambda t: None if t is None else t.data_ptr()
    out = torch.empty(B, T, H, device="cuda")
    if cell == "lstm":
        lib.call("fb_lstm_fwd", ctx.handle, ctx.stream, p(wi), p(wh), p(b), p(x), p(h0), p(c0), p(out), None, None, None, I, H, T, B)
    else:
        lib.call("fb_gru_fwd", ctx.handle, ctx.stream, p(wi), p(wh), p(b), p(x), p(h0), p(out), None, None, I, H, T, B)
    assert ctx.device_error() == 0
    zero = torch.zeros(B, H, device="cuda", dtype=torch.double)
    ref, _, _ = _reference(cell, wi.double(), wh.double(), b.double(), x.double(), zero if h0 is None else h0.double(), zero if c0 is None else c0.double())
    return out, ref


SIZES = [(48, 9, 40), (200, 20, 12), (512, 33, 6)]


@pytest.mark.parametrize("cell", ["lstm", "gru"])
@pytest.mark.parametrize("H,B,T", SIZES)
@pytest.mark.parametrize("scale", [1e-5, 1e-9, 1e-30])
def test_small_signals(cell, H, B, T, scale):
    """States of any size are held to 23 bits of the largest of their 64: relative to the outputs the error is that of ordinary ones."""
    g = torch.Generator(device="cuda").manual_seed(H)
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ng = 4 if cell == "lstm" else 3
    wi, wh, b, x = new(12, ng * H) / 4, new(H, ng * H) / H ** 0.5, torch.zeros(ng * H, device="cuda"), new(B, T, 12) * scale
    out, ref = _forward(cell, wi, wh, b, x, None)
    assert float((out.double() - ref).abs().max() / ref.abs().max()) < 5e-6


@pytest.mark.parametrize("H,B,T", SIZES)
@pytest.mark.parametrize("large", [1e3, 1e9, 1e30, float("inf")])
def test_a_large_initial_state(H, B, T, large):
    """A unit of a GRU far above the others, which do not read it; and one that saturates every gate, so that each state stays what it was."""
    g = torch.Generator(device="cuda").manual_seed(H)
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    wi, wh, b, x, h0 = new(12, 3 * H) / 4, new(H, 3 * H) / H ** 0.5, new(3 * H) * 0.1, new(B, T, 12), new(B, H)
    h0[::2, 7] = large
    if large < 1e38:
        wh0 = wh.clone()
        wh0[7] = 0.0
        out, ref = _forward("gru", wi, wh0, b, x, h0)
        others = [u for u in range(H) if u != 7]
        assert float((out.double() - ref)[:, :, others].abs().max()) < 5e-6
    wh[7] = wh[7].abs() + 1.0
    out, ref = _forward("gru", wi, wh, b, x, h0)
    if large >= 1e9:
        assert torch.equal(out[::2], h0[::2, None].expand(-1, T, -1))
    assert float((out.double() - ref)[1::2].abs().max()) < 5e-6


@pytest.mark.parametrize("cell", ["lstm", "gru"])
@pytest.mark.parametrize("H,B,T", SIZES)
@pytest.mark.parametrize("bad", [float("inf"), -float("inf"), float("nan")])
def test_weights_that_are_not_finite(cell, H, B, T, bad):
    """An infinite weight saturates the gates that it feeds and nothing else; what is finite in exact arithmetic is finite."""
    g = torch.Generator(device="cuda").manual_seed(H)
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ng = 4 if cell == "lstm" else 3
    wi, wh, b, x = new(12, ng * H) / 4, new(H, ng * H) / H ** 0.5, new(ng * H) * 0.1, new(B, T, 12)
    wh[3, 5], wh[H - 1, H + 40] = bad, bad
    out, ref = _forward(cell, wi, wh, b, x, new(B, H), new(B, H) if cell == "lstm" else None)
    assert torch.equal(torch.isfinite(out), torch.isfinite(ref)) and torch.equal(torch.isnan(out), torch.isnan(ref))
    fine = torch.isfinite(ref)
    assert float((out.double() - ref)[fine].abs().max()) < 5e-6


@pytest.mark.parametrize("cell", ["lstm", "gru"])
def test_gradients_that_are_not_finite_stay_in_their_column(cell):
    import fluxb200 as F
    from fluxb200 import lib
    gen = torch.Generator(device="cuda").manual_seed(0)
    H, B, T, I, ng = 128, 18, 12, 16, 4 if cell == "lstm" else 3
    new = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    ctx, wi, wh, bb, x = F.context(0), new(I, ng * H) * 0.2, new(H, ng * H) * 0.2, new(ng * H) * 0.2, new(B, T, I)
    p = lambda t: t.data_ptr()
    for bad in (float("inf"), float("nan")):
        dout = new(B, T, H)
        res = []
        for value in (1.0, bad):
            dout[4, T - 2, 9] = value
            n = getattr(lib.raw(), f"fb_{cell}_cache_bytes")(I, H, T, B) // 4
            cache, o = torch.empty(n, device="cuda"), torch.empty(B, T, H, device="cuda")
            g = [torch.empty_like(t) for t in (wi, wh, bb, x)]
            if cell == "lstm":
                lib.call("fb_lstm_fwd", ctx.handle, ctx.stream, p(wi), p(wh), p(bb), p(x), None, None, p(o), None, None, p(cache), I, H, T, B)
                lib.call("fb_lstm_bwd", ctx.handle, ctx.stream, p(wi), p(wh), p(x), None, None, p(o), p(cache), p(dout), None, None, *map(p, g), I, H, T, B)
            else:
                lib.call("fb_gru_fwd", ctx.handle, ctx.stream, p(wi), p(wh), p(bb), p(x), None, p(o), None, p(cache), I, H, T, B)
                lib.call("fb_gru_bwd", ctx.handle, ctx.stream, p(wi), p(wh), p(x), None, p(o), p(cache), p(dout), None, *map(p, g), I, H, T, B)
            assert ctx.device_error() == 0
            res.append(g[3].view(B, T, I).clone())
        others = [i for i in range(B) if i != 4]
        # (columns that share fragments with it are summed in Float32 instead of planes)
        assert float((res[0] - res[1])[others].abs().max()) < 2e-5 * float(res[0].abs().max())
        assert not bool(torch.isfinite(res[1][4, :T - 1]).any())


def _gradients(cell, wi, wh, b, x, dout):
    import fluxb200 as F
    from fluxb200 import lib
    ctx, (B, T, I), H = F.context(0), x.shape, wh.shape[0]
    p = lambda t: t.data_ptr()
    cache, o = torch.empty(getattr(lib.raw(), f"fb_{cell}_cache_bytes")(I, H, T, B) // 4, device="cuda"), torch.empty(B, T, H, device="cuda")
    g = [torch.empty_like(t) for t in (wi, wh, b, x)]
    if cell == "lstm":
        lib.call("fb_lstm_fwd", ctx.handle, ctx.stream, p(wi), p(wh), p(b), p(x), None, None, p(o), None, None, p(cache), I, H, T, B)
        lib.call("fb_lstm_bwd", ctx.handle, ctx.stream, p(wi), p(wh), p(x), None, None, p(o), p(cache), p(dout), None, None, *map(p, g), I, H, T, B)
    else:
        lib.call("fb_gru_fwd", ctx.handle, ctx.stream, p(wi), p(wh), p(b), p(x), None, p(o), None, p(cache), I, H, T, B)
        lib.call("fb_gru_bwd", ctx.handle, ctx.stream, p(wi), p(wh), p(x), None, p(o), p(cache), p(dout), None, *map(p, g), I, H, T, B)
    assert ctx.device_error() == 0
    return g


@pytest.mark.parametrize("cell", ["lstm", "gru"])
@pytest.mark.parametrize("H,B,T", [(400, 130, 4), (400, 130, 30), (512, 150, 3), (512, 70, 40)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_chunks_of_columns_do_not_meet(cell, H, B, T, bad):
    """Several chunks of columns per CTA.  A cotangent that is not finite at the last step sends the warps of its chunk through sums of
    very different length (25 groups of units: warp 0 alone has a fourth one): no column of another chunk changes a bit."""
    gen = torch.Generator(device="cuda").manual_seed(H + T)
    new = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    ng = 4 if cell == "lstm" else 3
    wi, wh, b, x, dout = new(16, ng * H) * 0.2, new(H, ng * H) / H ** 0.5, new(ng * H) * 0.1, new(B, T, 16), new(B, T, H)
    want = _gradients(cell, wi, wh, b, x, dout)[3].clone()
    for col in (0, 17, B - 1):
        held = dout[col, T - 1].clone()
        dout[col, T - 1, ::5] = bad
        got = _gradients(cell, wi, wh, b, x, dout)[3]
        dout[col, T - 1] = held
        others = [i for i in range(B) if i // 16 != col // 16]   # (chunks are of 8 or 16 columns)
        assert torch.equal(got[others], want[others])
        assert not bool(torch.isfinite(got[col, T - 1]).all())


@pytest.mark.parametrize("cell", ["lstm", "gru"])
@pytest.mark.parametrize("H,B,T", [(400, 130, 2), (400, 130, 5), (512, 150, 3), (496, 700, 4), (512, 70, 2)])
def test_chunks_of_columns_repeat_their_bits(cell, H, B, T):
    """The first step, which waits for nothing, and the last, which sends nothing, again and again; infinite weights of one group of units
    make the warp that owns it slower than the others.  Finite columns against float64: 2e-5 as above."""
    gen = torch.Generator(device="cuda").manual_seed(H + B)
    new = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    ng = 4 if cell == "lstm" else 3
    wi, wh, b, x, dout = new(12, ng * H) * 0.2, new(H, ng * H) / H ** 0.5, new(ng * H) * 0.1, new(B, T, 12), new(B, T, H)
    leaf = [t.double().requires_grad_() for t in (wi, wh, b, x)]
    zero = torch.zeros(B, H, device="cuda", dtype=torch.double)
    (_reference(cell, *leaf, zero, zero)[0] * dout.double()).sum().backward()
    first = [t.clone() for t in _gradients(cell, wi, wh, b, x, dout)]
    for got, want in zip(first, leaf):
        assert float((got.double() - want.grad).abs().max() / want.grad.abs().max()) < 2e-5
    for _ in range(8):
        assert all(torch.equal(a, c) for a, c in zip(_gradients(cell, wi, wh, b, x, dout), first))
    wh[20, 3] = float("inf")                                  # (the rows of the second group alone: its warp sums in Float32)
    slow = [t.clone() for t in _gradients(cell, wi, wh, b, x, dout)]
    for _ in range(8):
        assert all(torch.equal(torch.nan_to_num(a), torch.nan_to_num(c)) for a, c in zip(_gradients(cell, wi, wh, b, x, dout), slow))
