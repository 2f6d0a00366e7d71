"""GPU tests of the matmul kernels where their cuts fall: K ranges shared by a cluster, 16-wide tiles, remainders of the
64 x 64 and 128 x 256 tiles, rows that do not start on 16-byte boundaries.  Reference: the product in float64.

Tolerance: an FMA chain of K terms of N(0, 1) products is off by at most K * 2^-24 * sum|a b| / 2 and in practice by
sqrt(K) of it; the tensor-core path drops terms of 2^-22 and truncates while it accumulates (at most 2048 terms at a time).
3e-5 of the result's norm covers both; bf16 storage rounds the result to 2^-9."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import fluxb200 as F
    return F.context(0)


def _operands(ta, tb, m, n, k, pad, dtype):
    """Column-major op(A)[m, k] op(B)[k, n] as row-major torch views with `pad` extra values per row."""
    g = torch.Generator(device="cuda").manual_seed(m * 31 + n * 7 + k)
    ra, ca = (m, k) if ta else (k, m)
    rb, cb = (k, n) if tb else (n, k)
    A = torch.randn(ra, ca + pad, generator=g, device="cuda").to(dtype)
    B = torch.randn(rb, cb + pad, generator=g, device="cuda").to(dtype)
    a64, b64 = A[:, :ca].double(), B[:, :cb].double()
    ref = (b64.T if tb else b64) @ (a64.T if ta else a64)      # [n][m]
    return A, B, ref


# the FMA kernel: one row, 16-row and 16-column tiles and one past them, K of less than a stage, of several clusters, odd
# leading dimensions; the tensor-core kernel: K split over 2, 4 and 8 CTAs (with a ragged last part and two accumulation
# segments per part), pairs
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("m,n,k,pad", [(512, 1, 784, 0), (10, 16, 33, 1), (65, 17, 1, 0), (16, 300, 1000, 3), (33, 129, 260, 2),
                                       (520, 300, 1000, 0), (264, 140, 2100, 0), (516, 1030, 4100, 0), (1000, 1000, 9000, 0),
                                       (601, 515, 701, 0), (1003, 259, 2049, 1)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_gemm_f32_cuts(ctx, ta, tb, m, n, k, pad, accumulate):
    from fluxb200 import lib
    A, B, ref = _operands(ta, tb, m, n, k, pad, torch.float32)
    out = torch.ones(n, m + pad, device="cuda")
    lib.call("fb_gemm_f32", ctx.handle, ctx.stream, ta, tb, m, n, k, C.c_void_p(A.data_ptr()), A.shape[1], C.c_void_p(B.data_ptr()),
             B.shape[1], C.c_void_p(out.data_ptr()), m + pad, accumulate, 0)
    assert ctx.device_error() == 0
    err = (out[:, :m].double() - (1.0 if accumulate else 0.0) - ref).norm() / ref.norm()
    assert err < 3e-5, float(err)
    assert bool((out[:, m:] == 1.0).all())     # nothing is written between the rows


# few tiles and long K: K split over 8, 4 and 2 CTAs, whole tiles of one wave, pairs
@pytest.mark.parametrize("m,n,k,even", [(104, 1032, 12256, 745), (240, 736, 12624, 1023), (192, 104, 5760, 512), (64, 4096, 4096, 885),
                                        (512, 512, 16384, 1664), (1024, 1024, 16384, 1664), (1296, 2216, 1528, 1115), (5184, 512, 1216, 690),
                                        (672, 4288, 6008, 1664), (4096, 1024, 4096, 2048)])
def test_truncating_sums_are_no_longer_than_an_even_cut(ctx, m, n, k, even):
    """The tensor core truncates while it accumulates: 7.3e-9 of the result's norm per k-value of one accumulation (measured
    at 512 .. 2048 on N(0, 1) operands; its average of half a unit in the last place per add gives 1.5e-8).  `even` is the
    length that an even cut of all k-blocks over the SMs gives, between 512 and 1664 (2048 where whole tiles fill 3/4 of
    them)."""
    from fluxb200 import lib
    for ta, tb in ((0, 0), (0, 1)):
        A, B, ref = _operands(ta, tb, m, n, k, 0, torch.float32)
        out = torch.empty(n, m, device="cuda")
        lib.call("fb_gemm_f32", ctx.handle, ctx.stream, ta, tb, m, n, k, A.data_ptr(), A.shape[1], B.data_ptr(), B.shape[1], out.data_ptr(), m,
                 0, 0)
        err = float((out.double() - ref).norm() / ref.norm())
        assert err < 8.5e-9 * even, err


# tiles of several accumulation segments that meet in the workspace: pairs, one-CTA tiles, tiles shared by a cluster
@pytest.mark.parametrize("out_dim,in_dim,n", [(512, 1216, 5184), (10240, 3000, 200), (264, 9000, 520)])
@pytest.mark.parametrize("act", ["identity", "gelu_tanh"])
def test_epilogues_behind_parked_segments(ctx, out_dim, in_dim, n, act):
    from fluxb200 import lib
    g = torch.Generator(device="cuda").manual_seed(n)
    W = torch.randn(in_dim, out_dim, generator=g, device="cuda") / in_dim ** 0.5
    b, x = torch.randn(out_dim, generator=g, device="cuda"), torch.randn(n, in_dim, generator=g, device="cuda")
    y, z = torch.empty(n, out_dim, device="cuda"), torch.empty(n, out_dim, device="cuda")
    lib.call("fb_dense_fwd", ctx.handle, ctx.stream, lib.ACT[act], 0, W.data_ptr(), b.data_ptr(), x.data_ptr(), y.data_ptr(), z.data_ptr(),
             out_dim, in_dim, n)
    zr = x.double() @ W.double() + b.double()
    yr = zr if act == "identity" else torch.nn.functional.gelu(zr, approximate="tanh")
    assert ((z.double() - zr).norm() / zr.norm()) < 3e-5 and ((y.double() - yr).norm() / yr.norm()) < 3e-5
    before = y.clone()
    lib.call("fb_gemm_f32", ctx.handle, ctx.stream, 0, 0, out_dim, n, in_dim, W.data_ptr(), out_dim, x.data_ptr(), in_dim, y.data_ptr(), out_dim, 1, 0)
    ref = before.double() + zr - b.double()
    assert ((y.double() - ref).norm() / ref.norm()) < 3e-5 and ctx.device_error() == 0


def test_the_tensor_core_kernel_refuses_unaligned_results(ctx):
    from fluxb200 import lib
    A, B, _ = _operands(0, 0, 512, 512, 512, 0, torch.float32)
    out = torch.zeros(512, 513, device="cuda")
    for precision in ("3xtf32", "tf32", "3xtf32_pair"):
        with pytest.raises(lib.FluxB200Error):
            lib.call("fb_gemm_f32", ctx.handle, ctx.stream, 0, 0, 512, 512, 512, A.data_ptr(), 512, B.data_ptr(), 512, out.data_ptr(), 513, 0,
                     lib.PREC[precision])
    assert not bool(out.any())


def test_reserved_sms_keep_the_k_split(ctx):
    """With SMs left to communication kernels no clusters are used; 16 tiles of 1024 k-blocks still spread over the others
    (a whole tile each takes six times as long), and the results are those of a product."""
    from fluxb200 import lib
    m = n = 512
    A, B, ref = _operands(0, 0, m, n, 16384, 0, torch.float32)
    out = torch.empty(n, m, device="cuda")

    def product():
        lib.call("fb_gemm_f32", ctx.handle, ctx.stream, 0, 0, m, n, 16384, A.data_ptr(), m, B.data_ptr(), 16384, out.data_ptr(), m, 0, 0)

    def time_us():
        for _ in range(3):
            product()
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        for _ in range(10):
            product()
        end.record()
        torch.cuda.synchronize()
        return start.elapsed_time(end) * 100
    free = time_us()
    ctx.set_reserved_sms(8)
    try:
        reserved = time_us()
        assert ((out.double() - ref).norm() / ref.norm()) < 3e-5
    finally:
        ctx.set_reserved_sms(0)
    assert reserved < 3 * free, (reserved, free)


@pytest.mark.parametrize("rows", [17, 31])
@pytest.mark.parametrize("out_dim,in_dim", [(8192, 8192), (16384, 4096), (4096, 1024)])
def test_few_rows_go_to_the_faster_kernel(ctx, rows, out_dim, in_dim):
    """17 to 31 rows: the default precision takes no more than 1.3 times what the better of the two kernels takes (the FMA
    kernel needs twice the tensor cores' time at the largest of these sizes)."""
    from fluxb200 import lib
    A, B, ref = _operands(0, 0, out_dim, rows, in_dim, 0, torch.float32)
    out = torch.empty(rows, out_dim, device="cuda")

    def time_us(precision):
        def product():
            lib.call("fb_gemm_f32", ctx.handle, ctx.stream, 0, 0, out_dim, rows, in_dim, A.data_ptr(), out_dim, B.data_ptr(), in_dim,
                     out.data_ptr(), out_dim, 0, precision)
        for _ in range(3):
            product()
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        for _ in range(20):
            product()
        end.record()
        torch.cuda.synchronize()
        return start.elapsed_time(end) * 50
    fma, tc, default = time_us(lib.PREC["fp32_simt"]), time_us(lib.PREC["3xtf32"]), time_us(lib.PREC["default"])
    assert default < 1.3 * min(fma, tc), (fma, tc, default)
    assert ((out.double() - ref).norm() / ref.norm()) < 3e-5


# an odd leading dimension of one operand, of the result alone, and a start off the 16-byte boundary
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("m,n,k,lda,ldb,ldc,shift", [(1001, 1003, 1005, 0, 0, 0, 0), (512, 1024, 2048, 1, 0, 0, 0), (512, 1024, 2048, 0, 3, 0, 0),
                                                     (512, 1024, 2048, 0, 0, 2, 0), (1024, 512, 512, 0, 0, 0, 1), (4095, 33, 2049, 0, 0, 0, 0)])
def test_unaligned_products_keep_float32_sums(ctx, ta, tb, m, n, k, lda, ldb, ldc, shift):
    """The default precision computes them with Float32 FMAs: rounding to nearest, the errors of a sum of K terms add up as a
    random walk, sqrt(K) * 2^-24 of the result's norm with room to spare (3xTF32: truncated sums, 2^-22 terms left out);
    an infinite operand gives an infinite result."""
    from fluxb200 import lib
    g = torch.Generator(device="cuda").manual_seed(m + n + k)

    def mat(rows, cols, pad):
        flat = torch.randn(rows * (cols + pad) + 1, generator=g, device="cuda")
        return flat[shift:shift + rows * (cols + pad)].view(rows, cols + pad)
    (ra, ca), (rb, cb) = ((m, k) if ta else (k, m)), ((k, n) if tb else (n, k))
    A, B, out = mat(ra, ca, lda), mat(rb, cb, ldb), mat(n, m, ldc)

    def run():
        lib.call("fb_gemm_f32", ctx.handle, ctx.stream, ta, tb, m, n, k, A.data_ptr(), ca + lda, B.data_ptr(), cb + ldb, out.data_ptr(),
                 m + ldc, 0, 0)
        a, b = A[:, :ca].double(), B[:, :cb].double()
        return out[:, :m].double(), (b.T if tb else b) @ (a.T if ta else a)
    got, ref = run()
    err = float((got - ref).norm() / ref.norm())
    assert err < k ** 0.5 * 2.0 ** -24, err
    A[1, 2] = float("inf")
    got, ref = run()
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isinf(got), torch.isinf(ref))


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(512, 104, 784), (264, 200, 1000), (1000, 2048, 4096), (1024, 1024, 8200), (136, 8, 64), (520, 264, 64)])
@pytest.mark.parametrize("f32", [0, 1])
def test_gemm_bf16_cuts(ctx, ta, tb, m, n, k, f32):
    from fluxb200 import lib
    A, B, ref = _operands(ta, tb, m, n, k, 0, torch.bfloat16)
    for accumulate in (0, 1):
        out = torch.ones(n, m, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
        lib.call("fb_gemm_bf16", ctx.handle, ctx.stream, ta, tb, m, n, k, C.c_void_p(A.data_ptr()), A.shape[1], C.c_void_p(B.data_ptr()),
                 B.shape[1], C.c_void_p(out.data_ptr()), m, accumulate, f32)
        err = (out.double() - (1.0 if accumulate else 0.0) - ref).norm() / ref.norm()
        assert err < (3e-5 if f32 else 2.0 ** -9), float(err)
    assert ctx.device_error() == 0


@pytest.mark.parametrize("m,n,k", [(509, 104, 784), (77, 200, 64), (1021, 2048, 4096), (250, 300, 5000)])
@pytest.mark.parametrize("f32", [0, 1])
def test_gemm_bf16_ragged_rows(ctx, m, n, k, f32):
    """rows of the result that are no multiple of 8 long, in plain and shared tiles; the padding of a row stays as it is"""
    from fluxb200 import lib
    ld = (m + 7) // 8 * 8
    A, B, ref = _operands(0, 0, m, n, k, 0, torch.bfloat16)
    A = torch.nn.functional.pad(A, (0, ld - m))
    out = torch.full((n, ld), 3.0, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
    lib.call("fb_gemm_bf16", ctx.handle, ctx.stream, 0, 0, m, n, k, A.data_ptr(), ld, B.data_ptr(), B.shape[1], out.data_ptr(), ld, 0, f32)
    assert float((out[:, :m].double() - ref).norm() / ref.norm()) < (3e-5 if f32 else 2.0 ** -9)
    assert bool((out[:, m:] == 3.0).all()) and ctx.device_error() == 0


@pytest.mark.parametrize("act", ["identity", "relu", "gelu_tanh"])
@pytest.mark.parametrize("out_dim,in_dim,n", [(512, 784, 1), (10, 512, 100), (513, 300, 70), (512, 784, 1024), (1001, 520, 500)])
def test_dense_forward_epilogues_of_cut_tiles(ctx, act, out_dim, in_dim, n):
    """bias, activation and pre-activation store behind every way a tile is finished"""
    from fluxb200 import lib
    g = torch.Generator(device="cuda").manual_seed(out_dim + n)
    W = torch.randn(in_dim, out_dim, generator=g, device="cuda") / in_dim ** 0.5
    b = torch.randn(out_dim, generator=g, device="cuda")
    x = torch.randn(n, in_dim, generator=g, device="cuda")
    y, z = torch.empty(n, out_dim, device="cuda"), torch.empty(n, out_dim, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    lib.call("fb_dense_fwd", ctx.handle, ctx.stream, lib.ACT[act], 0, p(W), p(b), p(x), p(y), p(z), out_dim, in_dim, n)
    zr = x.double() @ W.double() + b.double()
    yr = {"identity": lambda v: v, "relu": torch.relu, "gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[act](zr)
    assert ((z.double() - zr).norm() / zr.norm()) < 3e-5
    assert ((y.double() - yr).norm() / yr.norm()) < 3e-5
    assert ctx.device_error() == 0


@pytest.mark.parametrize("m,n,k", [(512, 512, 32768), (1000, 2048, 4096), (1024, 5120, 2048)])
def test_split_products_on_several_streams(ctx, m, n, k):
    """Products that park segments or the parts of a cut last wave in memory of their own, on two streams and beside the
    replays of a graph on a third: every result is the serial one, bit for bit."""
    from fluxb200 import lib
    sets = []
    for i in range(3):
        g = torch.Generator(device="cuda").manual_seed(i)
        A, B = (torch.randn(k, d, generator=g, device="cuda") for d in (m, n))
        sets.append((A, B.T.contiguous(), torch.empty(n, m, device="cuda"), torch.empty(n, m, device="cuda")))

    def product(s, out):
        lib.call("fb_gemm_f32", ctx.handle, ctx.stream, 0, 0, m, n, k, s[0].data_ptr(), m, s[1].data_ptr(), k, out.data_ptr(), m, 0, 0)
    for s in sets:
        product(s, s[3])
    torch.cuda.synchronize()
    ref = sets[0][1].double() @ sets[0][0].double()
    assert ((sets[0][3].double() - ref).norm() / ref.norm()) < 3e-5
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        product(sets[2], sets[2][2])
        product(sets[2], sets[2][2])
    streams = [torch.cuda.Stream() for _ in range(3)]
    for _ in range(10):
        for s, st in zip(sets[:2], streams):
            with torch.cuda.stream(st):
                product(s, s[2])
                product(s, s[2])
        with torch.cuda.stream(streams[2]):
            graph.replay()
    torch.cuda.synchronize()
    for s in sets:
        assert torch.equal(s[2], s[3])
    assert ctx.device_error() == 0
