"""How far results are from FP64 where a product takes a route of its own: narrow
tiles, k slices, operands split inside the kernel.  None of them may round more
than whole 256-wide tiles, or k slices of them, of the same depth.

Each bound is the normwise error that those gave (U[-1, 1) operands, measured)
and 4% for the sample: the norm of N independent rounding errors varies by about
1/sqrt(2 N), at most 0.4% with the 2^16 elements or more of these outputs, between
inputs, and the error by 1 or 2% with their values."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
import ugemm_gb300 as ug  # noqa: E402

SAMPLE = 1.04


@pytest.fixture(scope="module", autouse=True)
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ug.build()
    ug.load()


def mat(r, c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand((r, c), device="cuda", generator=g) * 2 - 1


def rel(a, b):
    return float(torch.linalg.norm(a.double() - b) / torch.linalg.norm(b))


@pytest.mark.parametrize("prec", ["bf16x6", "bf16x9"])
@pytest.mark.parametrize("M,N,K,bound", [
    (256, 256, 256, 7.30e-8), (1024, 1024, 256, 7.29e-8), (128, 6000, 256, 7.29e-8),
    (512, 512, 512, 8.27e-8), (3648, 22, 38, 4.74e-8)])
def test_corrections_add_one_rounding(prec, M, N, K, bound):
    """Six accumulators of a 64-wide tile: the corrections are summed among
    themselves before they meet the main sum."""
    A, B = mat(M, K, M + K), mat(K, N, N)
    assert rel(ug.gemm(A, B, precision=prec), ug.ref64("N", "N", A, B)) < SAMPLE * bound


# deep k: as long sums as the slices of whole tiles would take
@pytest.mark.parametrize("prec,M,N,K,bound", [
    ("bf16x6", 1024, 1024, 1024, 8.73e-8), ("bf16x6", 256, 256, 1500, 1.13e-7),
    ("bf16x6", 2048, 2048, 2048, 1.16e-7), ("bf16x6", 1536, 2560, 4096, 1.25e-7),
    ("bf16x6", 2048, 2048, 8192, 2.04e-7), ("bf16x9", 2048, 2048, 4096, 1.26e-7),
    ("bf16x9", 128, 6000, 1024, 8.76e-8), ("fp16x3", 2048, 2048, 4096, 2.04e-7),
    ("fp16x3", 300, 4000, 1024, 1.35e-7), ("tf32x3", 2048, 2048, 4096, 3.36e-7)])
def test_sums_as_long_as_slices(prec, M, N, K, bound):
    A, B = mat(M, K, M + K), mat(K, N, N)
    assert rel(ug.gemm(A, B, precision=prec), ug.ref64("N", "N", A, B)) < SAMPLE * bound


@pytest.mark.parametrize("which,bound", [("A", 2.00e-7), ("B", 1.19e-7)])
def test_one_gradient(which, bound):
    M, N, K = 2048, 8192, 1024
    A, B, dC = mat(M, K, 1), mat(K, N, 2), mat(M, N, 3)
    out = torch.empty((M, K) if which == "A" else (K, N), device="cuda")
    ug.sgemm_backward("N", "N", M, N, K, 1.0, A, K, B, N, dC, N, 0.0, out if which == "A" else None,
                      K, 0.0, out if which == "B" else None, N, precision="bf16x6")
    ref = ug.ref64("N", "T", dC, B) if which == "A" else ug.ref64("T", "N", A, dC)
    assert rel(out, ref) < SAMPLE * bound


@pytest.mark.parametrize("prec,M,N,K,bound", [("bf16x6", 2048, 2048, 2048, 1.85e-7),
                                              ("bf16x9", 2048, 2048, 8192, 2.07e-7),
                                              ("bf16x6", 512, 512, 512, 1.93e-7)])
def test_plan_of_one_product(prec, M, N, K, bound):
    A, B, C = mat(M, K, 1), mat(K, N, 2), torch.empty((M, N), device="cuda")
    plan = ug.GroupedPlan([dict(ta="N", tb="N", M=M, N=N, K=K, alpha=1.0, beta=0.0, A=A, lda=K,
                                B=B, ldb=N, C=C, ldc=N)], precision=prec)
    plan.run()
    assert rel(C, ug.ref64("N", "N", A, B)) < SAMPLE * bound
    plan.close()


def test_convolution_layer():
    """U[0, 1) activations, He-normal weights, the output as its own gradient: a layer
    whose forward and weight gradient were three and two slices of 256-wide tiles."""
    cin, cout, n, batch = 128, 200, 13, 16
    st = ug.ConvStack([(cin, cout, n, n, 2)], batch, precision="bf16x6")
    g = torch.Generator(device="cuda").manual_seed(17)
    x, w = st.tensor(0, "x", (cin, batch, n, n)), st.tensor(0, "w", (cout, cin * 9))
    x.copy_(torch.rand(x.shape, device="cuda", generator=g))
    w.copy_(torch.randn(w.shape, device="cuda", generator=g) * (2.0 / (cin * 9)) ** 0.5)
    y = st.tensor(0, "y", (cout, batch * 49))
    st.run(ug.CONV_FORWARD)
    cols = torch.nn.functional.unfold(x.double().permute(1, 0, 2, 3).contiguous(), 3, padding=1,
                                      stride=2).permute(1, 0, 2).reshape(cin * 9, batch * 49)
    ref = w.double() @ cols
    assert rel(y, ref) < SAMPLE * 1.74e-7
    st.run(ug.CONV_BACKWARD)
    d = y.double()
    assert rel(st.tensor(0, "dw", (cout, cin * 9)), d @ cols.T) < SAMPLE * 3.83e-7
    dcol = (w.double().T @ d).reshape(cin * 9, batch, 49).permute(1, 0, 2)
    dx = torch.nn.functional.fold(dcol, (n, n), 3, padding=1, stride=2).permute(1, 0, 2, 3)
    assert rel(st.tensor(0, "dx", (cin, batch, n, n)), dx) < SAMPLE * 3.37e-7
    st.close()


@pytest.mark.parametrize("M,N,bound", [(8192, 16, 6.74e-8), (40000, 64, 7.9e-8)])
def test_gemv_partial_sums(M, N, bound):
    """Few columns: what adds the warps' sums rounds as much as the sums themselves."""
    At, x, y = mat(N, M, 3), mat(1, N, 4).reshape(-1), torch.zeros((M,), device="cuda")
    ug.sgemv("N", M, N, 1.0, At, M, x, 1, 0.0, y, 1)
    ref = torch.mv(At.double().T, x.double())
    assert rel(y, ref) < SAMPLE * bound


@pytest.mark.parametrize("prec", ["bf16x6", "bf16x9"])
@pytest.mark.parametrize("what,M,N,K,bound", [
    ("gemm", 1024, 1024, 672, 8.99e-8), ("gradient", 2048, 2048, 672, 8.98e-8),
    ("gradient", 1000, 3000, 928, 9.79e-8)])
def test_chunks_of_an_odd_depth(what, prec, M, N, K, bound):
    """21 and 29 stages: chunks of two and one of one, not 21 or 29 of one."""
    A, B = mat(M, K, 1), mat(K, N, 2)
    if what == "gemm":
        C = ug.gemm(A, B, precision=prec)
    else:  # C as the gradient of X in Y = X W, A that of Y
        C, W = torch.empty((M, N), device="cuda"), B.t().contiguous()
        ug.sgemm_backward("N", "N", M, K, N, 1.0, 0, N, W, K, A, K, 0.0, C, N, 0.0, None, K,
                          precision=prec)
    assert rel(C, ug.ref64("N", "N", A, B)) < SAMPLE * bound
