"""GPU tests of the one-launch recurrences at the edges of their cuts: one unit, one column, one step; hidden sizes and batches
just off the 8 / 16-unit and 4 / 8 / 16-column tiles; hidden sizes whose unit groups leave one batch group for several
chunks of columns; rows of several 512-wide pieces.  Oracle in float64; tolerances as in the recurrent tests of
test_gpu_kernels.py (1e-4 of the largest value, 2e-4 for gradients: two chained reductions)."""
import numpy as np
import pytest

import flux_oracle as O
from util import close

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1, 1), (2, 1, 3, 1), (5, 15, 2, 17), (4, 17, 4, 33), (8, 61, 3, 4), (6, 200, 3, 20), (3, 339, 2, 9), (4, 520, 2, 40),
          (3, 772, 2, 70), (2, 1030, 2, 35)]


@pytest.mark.parametrize("cell", ["lstm", "gru"])
@pytest.mark.parametrize("I,H,T,B", SHAPES)
def test_sequence_kernels(cell, I, H, T, B):
    import fluxb200 as F
    rng = np.random.default_rng(I + H + T + B)
    ng = 4 if cell == "lstm" else 3
    Wi, Wh = O.glorot_uniform(rng, ng * H, I), O.glorot_uniform(rng, ng * H, H)
    b = (rng.normal(size=ng * H) * 0.1).astype(np.float32)
    x = rng.normal(size=(I, T, B)).astype(np.float32)
    rnn = (F.LSTM if cell == "lstm" else F.GRU)(Wi, Wh, b.copy())
    xg = F.gpu(x)
    scan = O.lstm_scan_fwd if cell == "lstm" else O.gru_scan_fwd
    back = O.lstm_scan_bwd if cell == "lstm" else O.gru_scan_bwd
    a64 = [v.astype(np.float64) for v in (Wi, Wh, b, x)]
    ref = scan(*a64)[0]
    close(F.cpu(rnn(xg)), ref, name="out")
    # a NaN in one sample's input stays in that sample
    if B > 1 and T > 1:
        xn = x.copy()
        xn[0, 0, B - 1] = np.nan
        yn = F.cpu(rnn(F.gpu(xn)))
        assert np.isnan(yn[:, :, B - 1]).all()
        close(yn[:, :, :B - 1], ref[:, :, :B - 1], name="others")
    _, (g,) = F.withgradient(lambda m: F.sum_abs2(m(xg)), rnn)
    rWi, rWh, rb, _ = back(*a64, O.sum_abs2_bwd(ref))
    tol = dict(rtol=2e-4, atol_scale=2e-4)
    c = g["cell"]
    close(F.cpu(c["Wi"]), rWi, name="dWi", **tol)
    close(F.cpu(c["Wh"]), rWh, name="dWh", **tol)
    close(F.cpu(c["bias" if cell == "lstm" else "b"]), rb, name="db", **tol)
    assert F.context().device_error() == 0


# (a CTA walks several chunks of columns for many steps; hidden sizes beyond 512 that are no multiple of 4: scalar loads in
# several 512-wide pieces; three chunks of a small layer)
LONG = [("lstm", 3, 772, 40, 70), ("gru", 3, 772, 40, 70), ("gru", 5, 515, 30, 40), ("lstm", 4, 530, 30, 33), ("lstm", 6, 200, 60, 300),
        ("gru", 6, 203, 60, 300)]


def _rnn(cell, I, H, T, B):
    import fluxb200 as F
    rng = np.random.default_rng(I + H + T + B)
    ng = 4 if cell == "lstm" else 3
    Wi, Wh = O.glorot_uniform(rng, ng * H, I), O.glorot_uniform(rng, ng * H, H)
    b = (rng.normal(size=ng * H) * 0.1).astype(np.float32)
    x = rng.normal(size=(I, T, B)).astype(np.float32)
    state = tuple(rng.normal(size=(H, B)).astype(np.float32) for _ in range(2 if cell == "lstm" else 1))
    return (F.LSTM if cell == "lstm" else F.GRU)(Wi, Wh, b.copy()), (Wi, Wh, b, x), state


def _autograd(cell, arrays, state, out):
    """dWi, dWh, db of sum(abs2, out) in float64 (the oracle's reverse sweeps start from zero states)."""
    import torch
    Wi, Wh, b = (torch.tensor(v, requires_grad=True) for v in arrays[:3])
    x, h, c = torch.tensor(arrays[3]), torch.tensor(state[0]), torch.tensor(state[-1])
    total, worst = 0.0, 0.0
    for t in range(x.shape[1]):
        if cell == "lstm":
            i, f, g, o = (Wi @ x[:, t] + Wh @ h + b[:, None]).chunk(4)
            c = torch.sigmoid(f) * c + torch.sigmoid(i) * torch.tanh(g)
            h = torch.sigmoid(o) * torch.tanh(c)
        else:
            gx, gh = (Wi @ x[:, t] + b[:, None]).chunk(3), (Wh @ h).chunk(3)
            r, z = torch.sigmoid(gx[0] + gh[0]), torch.sigmoid(gx[1] + gh[1])
            h = (1 - z) * torch.tanh(gx[2] + r * gh[2]) + z * h
        total = total + (h * h).sum()
        worst = max(worst, float((h.detach() - torch.tensor(out[:, t])).abs().max()))
    assert worst < 1e-10      # the same recurrence as the oracle's
    total.backward()
    return [v.grad.numpy() for v in (Wi, Wh, b)]


@pytest.mark.parametrize("cell,I,H,T,B", LONG)
def test_long_sequences_with_initial_state(cell, I, H, T, B):
    import fluxb200 as F
    rnn, arrays, state = _rnn(cell, I, H, T, B)
    xg, sg = F.gpu(arrays[3]), tuple(F.gpu(s) for s in state)
    start = sg if cell == "lstm" else sg[0]
    a64, s64 = [v.astype(np.float64) for v in arrays], [v.astype(np.float64) for v in state]
    ref = (O.lstm_scan_fwd if cell == "lstm" else O.gru_scan_fwd)(*a64, *s64)[0]
    close(F.cpu(rnn(xg, start)), ref, name="out")
    _, (g,) = F.withgradient(lambda m: F.sum_abs2(m(xg, start)), rnn)
    grads = _autograd(cell, a64, s64, ref)
    # two chained reductions as above, over T * B columns
    tol = dict(rtol=2e-4, atol_scale=2e-4)
    c = g["cell"]
    close(F.cpu(c["Wi"]), grads[0], name="dWi", **tol)
    close(F.cpu(c["Wh"]), grads[1], name="dWh", **tol)
    close(F.cpu(c["bias" if cell == "lstm" else "b"]), grads[2], name="db", **tol)
    assert F.context().device_error() == 0


@pytest.mark.parametrize("cell,I,H,T,B", [("lstm", 64, 512, 24, 64), ("gru", 17, 203, 40, 90)])
def test_captured_sequences_replay_like_eager_calls(cell, I, H, T, B):
    """Forward and backward pass recorded into graphs and replayed on two streams at once (each wants more than half of the
    SMs): bit for bit the eager results."""
    import torch

    import fluxb200 as F
    from fluxb200 import lib
    ctx, sets = F.context(), []
    for i in range(2):
        _, (Wi, Wh, b, x), _ = _rnn(cell, I, H, T + i, B)
        arrays = [F.gpu(v) for v in (Wi, Wh, b, x)]
        steps = T + i
        cache = torch.empty(getattr(lib.raw(), f"fb_{cell}_cache_bytes")(I, H, steps, B) // 4, device="cuda")
        out, dout = F.empty((H, steps, B)), F.gpu(np.random.default_rng(i).normal(size=(H, steps, B)).astype(np.float32))
        grads = [F.empty(Wi.shape), F.empty(Wh.shape), F.empty(x.shape)]

        def run(arrays=arrays, cache=cache, out=out, dout=dout, grads=grads, steps=steps):
            Wi, Wh, b, x = (v.ptr for v in arrays)
            none, dims = (None,) * 2, (I, H, steps, B)
            if cell == "lstm":
                lib.call("fb_lstm_fwd", ctx.handle, ctx.stream, Wi, Wh, b, x, *none, out.ptr, *none, cache.data_ptr(), *dims)
                lib.call("fb_lstm_bwd", ctx.handle, ctx.stream, Wi, Wh, x, *none, out.ptr, cache.data_ptr(), dout.ptr, *none, grads[0].ptr,
                         grads[1].ptr, None, grads[2].ptr, *dims)
            else:
                lib.call("fb_gru_fwd", ctx.handle, ctx.stream, Wi, Wh, b, x, None, out.ptr, None, cache.data_ptr(), *dims)
                lib.call("fb_gru_bwd", ctx.handle, ctx.stream, Wi, Wh, x, None, out.ptr, cache.data_ptr(), dout.ptr, None, grads[0].ptr,
                         grads[1].ptr, None, grads[2].ptr, *dims)
        run()
        eager = [v.t.clone() for v in [out] + grads]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run()
        for v in [out] + grads:
            v.t.zero_()
        sets.append((graph, [out] + grads, eager, arrays, cache, dout))
    streams = [torch.cuda.Stream() for _ in sets]
    torch.cuda.synchronize()
    for _ in range(5):
        for (graph, *_), st in zip(sets, streams):
            with torch.cuda.stream(st):
                graph.replay()
    torch.cuda.synchronize()
    for _, results, eager, *_ in sets:
        assert all(torch.equal(a.t, b) for a, b in zip(results, eager))
    assert ctx.device_error() == 0
