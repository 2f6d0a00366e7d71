"""GPU test of two host threads, each with a context and a stream of its own, whose calls run the same kernels with different amounts of
shared memory: neither disturbs the other's launches."""
import ctypes as C
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _batchnorm(lib, ctx, stream, s, c, n):
    x = torch.randn(s * c * n, device="cuda")
    y, v = torch.empty_like(x), [torch.ones(c, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    return lambda: lib.call("fb_batchnorm_fwd_train", ctx, stream, x.data_ptr(), v[0].data_ptr(), v[1].data_ptr(), None, None, y.data_ptr(),
                            v[2].data_ptr(), v[3].data_ptr(), s, c, n, 1e-5, 0.1, 0, 0)


def _layernorm(lib, ctx, stream, d, n):
    x, dy = torch.randn(n * d, device="cuda"), torch.randn(n * d, device="cuda")
    dx, g, dg = torch.empty_like(x), torch.ones(d, device="cuda"), torch.empty(2 * d, device="cuda")
    m = torch.ones(n, device="cuda")
    torch.cuda.synchronize()
    return lambda: lib.call("fb_layernorm_bwd", ctx, stream, x.data_ptr(), g.data_ptr(), g.data_ptr(), m.data_ptr(), m.data_ptr(), dy.data_ptr(),
                            dx.data_ptr(), dg.data_ptr(), dg[d:].data_ptr(), d, n, 0)


@pytest.mark.parametrize("make,large,small", [(_batchnorm, (25600, 2, 2), (12544, 2, 2)), (_layernorm, (4096, 64), (2304, 64))])
def test_shared_memory_of_two_threads(make, large, small):
    import fluxb200  # noqa: F401
    from fluxb200 import lib
    errors = []

    def work(args):
        try:
            torch.cuda.set_device(0)
            h = C.c_void_p()
            lib.call("fb_ctx_create", 0, C.byref(h))
            stream = torch.cuda.Stream()
            step = make(lib, h.value, stream.cuda_stream, *args)
            start.wait()
            for _ in range(4000):
                step()
            stream.synchronize()
            lib.call("fb_ctx_destroy", h.value)
        except Exception as e:   # noqa: BLE001  (reported by the main thread)
            errors.append(e)
    start = threading.Barrier(2, timeout=60)
    threads = [threading.Thread(target=work, args=(a,)) for a in (large, small)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_an_error_is_reported_once():
    """A runtime call that fails (here: a wait inside a capture) is the error of the entry point that made it, not of the next one."""
    import fluxb200 as F
    from fluxb200 import lib
    ctx = F.context(0)
    x, y, m, r = torch.randn(64 * 10, device="cuda"), torch.empty(640, device="cuda"), torch.empty(10, device="cuda"), torch.empty(10, device="cuda")
    out = torch.zeros(1, dtype=torch.int32).pin_memory()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graph.capture_begin(capture_error_mode="relaxed")
        status = lib.raw().fb_device_error(ctx.handle, side.cuda_stream, C.cast(out.data_ptr(), C.POINTER(C.c_int32)))
    after = lib.raw().fb_layernorm_fwd(ctx.handle, torch.cuda.default_stream().cuda_stream, x.data_ptr(), None, None, y.data_ptr(), m.data_ptr(), r.data_ptr(), 64, 10,
                                       1e-5, 0)
    with torch.cuda.stream(side):
        try:
            graph.capture_end()
        except RuntimeError:
            pass
    torch.cuda.synchronize()
    assert status != 0 and after == 0, (status, after)
    assert torch.isfinite(y).all() and ctx.device_error() == 0
