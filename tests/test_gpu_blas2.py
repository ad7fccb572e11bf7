"""GPU SAXPY / SGEMV against the reference's saxpy_cpu / sgemv_cpu golden
outputs (ugemm.h:86-160) and against FP64 at larger sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
import ugemm_gb300 as ug  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ug.build()
    ug.load()


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def test_saxpy_golden(golden):
    for name in [c for c in golden["cases"] if str(c).startswith("axpy/")]:
        g = lambda k: golden[f"{name}/{k}"]  # noqa: E731
        n, incx, incy = (int(v) for v in g("meta"))
        y = dev(g("y"))
        ug.saxpy(n, 0.75, dev(g("x")), incx, y, incy)
        torch.cuda.synchronize()
        np.testing.assert_allclose(y.cpu().numpy(), g("out"), rtol=0, atol=2e-7)


def test_sgemv_golden(golden):
    for name in [c for c in golden["cases"] if str(c).startswith("gemv/")]:
        g = lambda k: golden[f"{name}/{k}"]  # noqa: E731
        M, N, lda, inc = (int(v) for v in g("meta"))
        y = dev(g("y"))
        ug.sgemv(bytes(g("flags")).decode(), M, N, 1.5, dev(g("A")), lda, dev(g("x")), inc, 0.5, y,
                 inc)
        torch.cuda.synchronize()
        ref = g("out")
        assert np.abs(y.cpu().numpy() - ref).max() / np.abs(ref).max() < 1e-5, name


@pytest.mark.parametrize("trans", ["N", "T"])
def test_sgemv_large_vs_fp64(trans):
    M, N = 5000, 3001
    lda = (M if trans == "N" else N) + 3
    cols = N if trans == "N" else M
    A = torch.rand((cols, lda), device="cuda") * 2 - 1   # column-major: one column per row of storage
    x = torch.rand(N, device="cuda") * 2 - 1
    y0 = torch.rand(M, device="cuda") * 2 - 1
    y = y0.clone()
    ug.sgemv(trans, M, N, 1.5, A, lda, x, 1, 0.5, y, 1)
    torch.cuda.synchronize()
    Am = A[:, :M].double().T if trans == "N" else A[:, :N].double()  # M x N
    ref = 1.5 * (Am @ x.double()) + 0.5 * y0.double()
    assert float(torch.linalg.norm(y.double() - ref) / torch.linalg.norm(ref)) < 2e-6


def test_saxpy_large_and_strided():
    n = (1 << 22) + 3
    x = torch.rand(n, device="cuda")
    y = torch.rand(n, device="cuda")
    ref = y.double() + 0.25 * x.double()
    ug.saxpy(n, 0.25, x, 1, y, 1)
    torch.cuda.synchronize()
    assert float((y.double() - ref).abs().max()) < 1e-6
    xs = torch.rand(3 * 1000, device="cuda")
    ys = torch.rand(2 * 1000, device="cuda")
    ref = ys.clone()
    ref[::2] += 2.0 * xs[::3]
    ug.saxpy(1000, 2.0, xs, 3, ys, 2)
    torch.cuda.synchronize()
    assert torch.allclose(ys, ref, atol=1e-6)


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("M,N,pad,off", [(512, 512, 0, 0), (516, 4097, 0, 0), (2436, 1025, 4, 0),
                                         (1, 9000, 0, 0), (31, 511, 1, 0), (5000, 2049, 3, 1),
                                         (640, 8200, 0, 1)])
def test_gemv_vector_widths_and_shared_columns(trans, M, N, pad, off):
    """Aligned and unaligned columns, one and several warps (or a cluster) per
    output.  FP32 sums of N products: within sqrt(N) 2^-24 ~ 6e-6 / 1e3 of FP64
    normwise; 2e-6 is the suite's bound."""
    rows, cols = (M, N) if trans == "N" else (N, M)   # column-major rows x cols
    lda = rows + pad
    g = torch.Generator(device="cuda").manual_seed(M + N)
    buf = torch.rand((cols * lda + 4,), device="cuda", generator=g) - 0.5
    A = buf[off:off + cols * lda].view(cols, lda)[:, :rows]
    x = torch.rand((N,), device="cuda", generator=g) - 0.5
    y = torch.rand((2 * M,), device="cuda", generator=g)
    a64 = A.double().T if trans == "N" else A.double()
    ref = 1.5 * (a64 @ x.double()) + 0.5 * y[::2].double()
    odd = y[1::2].clone()
    ug.sgemv(trans, M, N, 1.5, A.data_ptr(), lda, x, 1, 0.5, y, 2)
    torch.cuda.synchronize()
    assert float(torch.linalg.norm(y[::2].double() - ref) / torch.linalg.norm(ref)) < 2e-6
    assert torch.equal(y[1::2], odd)


def graph_us(f, n=20):
    """Microseconds a call of f takes on the device, in a graph of n."""
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    f()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        for _ in range(n):
            f()
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    best = 1e9
    for _ in range(8):
        e[0].record()
        g.replay()
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]))
    return best * 1000 / n


def gemv_us(trans, M, N, pad):
    lda, cols = (M + pad, N) if trans == "N" else (N + pad, M)
    A = torch.rand((lda * cols,), device="cuda")
    x, y = torch.rand((N,), device="cuda"), torch.zeros((M,), device="cuda")
    return graph_us(lambda: ug.sgemv(trans, M, N, 1.0, A, lda, x, 1, 0.0, y, 1))


def test_gemv_time_follows_the_size():
    """Blocks and warps that share an output must not cost more than they bring:
    unaligned columns in four-byte loads take less than twice the 16-byte ones (2.5
    times in clusters of eight), and 2000 short outputs no longer than 2600 (1.7
    times in eight warps each; 1.35 leaves room for the clock)."""
    assert gemv_us("N", 16384, 1024, 1) < 2 * gemv_us("N", 16384, 1024, 0)
    assert gemv_us("T", 2000, 100, 0) < 1.35 * gemv_us("T", 2600, 100, 0)


@pytest.mark.parametrize("M,N", [(1, 1), (127, 8), (129, 3), (2432 * 128 + 4, 5), (2432 * 128 + 5, 8),
                                 (33, 9), (9728, 96), (9732, 97), (19457, 31), (19456, 256),
                                 (78000, 17), (77825, 255), (300, 257), (1, 256)])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_gemv_few_columns(M, N, pad):
    """Threads with rows to themselves, and blocks of four to sixteen warps: the edges of
    each, strided vectors, y updated or (NaN in it) not read.  The products' rounding and
    a sum of N: within 2e-6 normwise, as elsewhere."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    lda, incx, incy = M + pad, 1 + pad % 3, 2
    A = torch.rand((N, lda), device="cuda", generator=g) * 2 - 1
    x = torch.rand((N * incx,), device="cuda", generator=g) + 0.5
    y = torch.rand((M * incy,), device="cuda", generator=g)
    ref = A[:, :M].double().T @ x[::incx].double()
    z, old = torch.full_like(y, float("nan")), y.clone()
    ug.sgemv("N", M, N, 1.5, A, lda, x, incx, 0.5, y, incy)
    ug.sgemv("N", M, N, 1.0, A, lda, x, incx, 0.0, z, incy)
    torch.cuda.synchronize()
    assert float(torch.linalg.norm(z[::incy].double() - ref) / torch.linalg.norm(ref)) < 2e-6
    want = 1.5 * ref + 0.5 * old[::incy].double()
    assert float(torch.linalg.norm(y[::incy].double() - want) / torch.linalg.norm(want)) < 2e-6
    assert torch.equal(y[1::incy], old[1::incy]) and bool(torch.isnan(z[1::incy]).all())


def test_gemv_time_of_few_columns():
    """One column is no more than a saxpy of as many elements (with eight warps to 32
    rows 6 times that; 3 leaves room), and loads in flight do not cost the warps that
    short columns live by: aligned ones take no longer than others (1.2 times with eight
    16-byte loads), and 96 floats in four-byte loads 1.1 times the aligned ones (1.45 with
    eight in flight)."""
    x, y = torch.rand((1000000,), device="cuda"), torch.rand((1000000,), device="cuda")
    assert gemv_us("N", 1000000, 1, 0) < 3 * graph_us(lambda: ug.saxpy(1000000, 0.5, x, 1, y, 1))
    assert gemv_us("T", 144896, 416, 0) < 1.1 * gemv_us("T", 144896, 416, 1)
    assert gemv_us("T", 94016, 96, 1) < 1.28 * gemv_us("T", 94016, 96, 0)


@pytest.mark.parametrize("trans,M,N", [("T", 16384, 1024), ("N", 30000, 500)])
def test_gemv_matrix_stays_in_l2(trans, M, N):
    """A matrix half as large as L2 is there for the next call: aligned columns are read no
    more slowly than unaligned ones (1.4 and 1.5 times when evicted first)."""
    A = [torch.rand((M * N + 4,), device="cuda")[i:i + M * N] for i in (0, 1)]
    x, y = torch.rand((N,), device="cuda"), torch.zeros((M,), device="cuda")
    us = [graph_us(lambda: ug.sgemv(trans, M, N, 1.0, a, M if trans == "N" else N, x, 1, 0.0, y, 1))
          for a in A]
    assert us[0] < 1.15 * us[1]
