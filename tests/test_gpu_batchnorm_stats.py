"""GPU tests of BatchNorm's batch statistics: values that are not finite, and inputs whose mean is far from zero.  Reference: float64."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
# (s, c, n): one CTA and clusters of 2 to 8 per channel, a value a thread, pieces of four, channels that do not fit shared memory, fewer
# samples than CTAs of a full cluster
SHAPES = [(1, 5, 40), (49, 6, 64), (1024, 8, 16), (1024, 40, 128), (784, 3, 33), (50176, 2, 16), (12544, 3, 256), (25600, 3, 1),
          (25600, 3, 2), (50176, 2, 3), (50175, 2, 2), (51200, 2, 1), (51204, 2, 1)]


@pytest.fixture(scope="module")
def ctx():
    import fluxb200 as F
    return F.context(0)


def _p(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def _forward(ctx, x, s, c, n):
    from fluxb200 import lib
    y, gamma, beta = torch.empty_like(x), torch.ones(c, device="cuda"), torch.zeros(c, device="cuda")
    rm, rv, sm, sr = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda"), torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    lib.call("fb_batchnorm_fwd_train", ctx.handle, ctx.stream, _p(x), _p(gamma), _p(beta), _p(rm), _p(rv), _p(y), _p(sm), _p(sr), s, c, n, 1e-5, 0.25, 0, 1)
    assert ctx.device_error() == 0
    return y, rm, rv, sm, sr


@pytest.mark.parametrize("s,c,n", SHAPES)
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_values_that_are_not_finite(ctx, s, c, n, bad):
    """They show in everything of their channel, the running variance among it, and in no other channel."""
    g = torch.Generator(device="cuda").manual_seed(s + n)
    x = torch.randn(n, c, s, generator=g, device="cuda")
    want = torch.zeros(c, dtype=torch.bool, device="cuda")
    want[1] = True
    for at in ((0, 0), (n - 1, s - 1), (n // 2, s // 3)):      # the channel's first value, its last, one in between
        x1 = x.clone()
        x1[at[0], 1, at[1]] = bad
        y, rm, rv, sm, sr = _forward(ctx, x1, s, c, n)
        for t in (rm, sm):
            assert torch.equal(~torch.isfinite(t), want)
        assert torch.equal(torch.isnan(rv), want) and torch.equal(torch.isnan(sr), want)
        assert torch.equal(torch.isnan(y).amax(dim=(0, 2)), want) and bool(torch.isnan(y[:, 1]).all())


@pytest.mark.parametrize("s,c,n", SHAPES + [(64, 4, 3000)])
@pytest.mark.parametrize("ratio", [0, 30, 1000])
def test_variance_of_values_far_from_zero(ctx, s, c, n, ratio):
    """mean / std = ratio, and a channel's first value, or the first of every sample (a zero border), far from all others.  A thread's
    sums of up to k values cancel by at most k of their own variance, 2^-24 each, with k <= 256; a deviation from a mean of
    `ratio` is off by the mean's own rounding, ratio 2^-24, which is uncorrelated between threads.  So 256 x 2^-24 = 1.5e-5,
    and 2 ratio 2^-24 (1.2e-4 at 1000)."""
    g = torch.Generator(device="cuda").manual_seed(s + n + ratio)
    for border in (0, 1, 2):
        x = torch.randn(n, c, s, generator=g, device="cuda") + ratio
        if border == 1:
            x[0, :, 0] = 0.0
        elif border == 2:
            x[:, :, 0] = 0.0
        y, rm, rv, sm, sr = _forward(ctx, x, s, c, n)
        v = x.double().transpose(0, 1).reshape(c, -1)
        var = v.var(dim=1, unbiased=False)
        tol = 1.5e-5 + 2 * ratio * 2.0 ** -24
        cnt = s * n
        for got, want in ((rv, 0.75 + 0.25 * var * cnt / (cnt - 1)), (sr, (var + 1e-5).rsqrt())):
            assert float(((got.double() - want) / want).abs().max()) < tol, border
        assert float((sm.double() - v.mean(dim=1)).abs().max()) <= 2.0 ** -21 * max(ratio, 1)


@pytest.mark.parametrize("s,c,n", [(256, 207, 24), (256, 300, 16), (64, 600, 64), (63, 170, 96), (192, 400, 20), (255, 200, 24), (1, 900, 4096),
                                   (196, 37, 85), (149, 144, 47), (256, 16, 184), (799, 38, 22), (469, 27, 96), (196, 74, 41)])
def test_channels_that_just_fit_without_asking_for_shared_memory(ctx, s, c, n):
    """Copies of 48 KB (and others near it) beside the kernel's own shared memory, alone and in clusters of two to eight.  Statistics of at most
    47 K ordinary values in Float32: 2e-6."""
    g = torch.Generator(device="cuda").manual_seed(s + c + n)
    x = torch.randn(n, c, s, generator=g, device="cuda")
    y, rm, rv, sm, sr = _forward(ctx, x, s, c, n)
    ref = x.double()
    mean, var = ref.mean((0, 2)), ref.var((0, 2), unbiased=False)
    want = (ref - mean[None, :, None]) / (var + 1e-5).sqrt()[None, :, None]
    assert float((y.double() - want).norm() / want.norm()) < 2e-6
    assert float((sm.double() - mean).abs().max()) < 2e-6 and float((rv.double() - (0.75 + 0.25 * ref.var((0, 2)))).abs().max()) < 2e-6
