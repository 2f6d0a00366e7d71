"""The one-pass update of bf16 parameters against the Float32 update between two casts: same rule, same roundings."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,shift", [([1], 0), ([3, 0, 8192], 0), ([8193, 5, 40000, 16383], 1), ([17] * 40, 0)])
def test_adam_bf16(counts, shift):
    """shift = 1: gradients and parameters that start 2 bytes past an 8-byte boundary; 40 leaves take two launches."""
    import fluxb200 as F
    from fluxb200 import lib
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(counts))
    ctx = F.context()
    arr = C.c_void_p * len(counts)

    def table(ts):
        return arr(*[t.data_ptr() for t in ts])

    def f32(scale):
        return [torch.randn(n, device="cuda", generator=g) * scale for n in counts]

    w, m = f32(1.0), f32(1e-3)
    v = [t.abs() * 1e-6 + 1e-8 for t in f32(1.0)]
    grad = [torch.empty(n + 4, device="cuda", dtype=torch.bfloat16)[shift:shift + n].copy_(t) for n, t in zip(counts, f32(1e-2))]
    low = [torch.empty(n + 4, device="cuda", dtype=torch.bfloat16)[shift:shift + n] for n in counts]
    w2, m2, v2, wide = [t.clone() for t in w], [t.clone() for t in m], [t.clone() for t in v], [t.float() for t in grad]
    cnt = (C.c_int64 * len(counts))(*counts)
    tail = (cnt, 1e-3, 0.9, 0.999, 1e-8, 0.81, 0.998, 0.5)
    lib.call("fb_adam_step_bf16", ctx.handle, ctx.stream, len(counts), table(low), table(w), table(grad), table(m), table(v), *tail)
    lib.call("fb_adam_step", ctx.handle, ctx.stream, len(counts), table(w2), table(wide), table(m2), table(v2), *tail)
    for a, b in zip(w + m + v, w2 + m2 + v2):
        # the compilers of the two kernels may contract a product and a sum differently: two roundings of 2^-24
        torch.testing.assert_close(a, b, rtol=2.4e-7, atol=1e-12)
    for a, b in zip(low, w):
        assert torch.equal(a, b.bfloat16())
