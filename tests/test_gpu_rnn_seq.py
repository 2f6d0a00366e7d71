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
