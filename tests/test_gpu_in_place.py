"""Products written into their own operands in the split forms: a launch on pieces has
read all operands before it writes, and launches that split them inside the kernel, which
read while other tiles are written, are not taken there.  Within 2e-6 of FP64."""
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


def mat(r, c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.rand((r, c), device="cuda", generator=g) * 2 - 1) / c ** 0.5


def rel(a, b):
    return float(torch.linalg.norm(a.double() - b) / torch.linalg.norm(b))


@pytest.mark.parametrize("prec", ["bf16x6", "bf16x9", "fp16x3", "tf32x3"])
@pytest.mark.parametrize("into", ["A", "B", "next"])
def test_group_into_its_operands(prec, into):
    """60 products of 500 x 256 x 256 (or 256 x 500 x 256), C over A, over B, or over the
    A of the group's next product."""
    M, N, K = (256, 500, 256) if into == "B" else (500, 256, 256)
    A = [mat(M, K, i) for i in range(60)]
    B = [mat(K, N, 100 + i) for i in range(60)]
    C = B if into == "B" else A if into == "A" else A[1:] + A[:1]
    refs = [a.double() @ b.double() for a, b in zip(A, B)]
    p = ug.GroupedPlan([dict(ta="N", tb="N", M=M, N=N, K=K, alpha=1.0, beta=0.0, A=a, lda=K, B=b,
                             ldb=N, C=c, ldc=N) for a, b, c in zip(A, B, C)], precision=prec)
    assert p.config["fused"] == 0
    p.run()
    p.check()
    for c, ref in zip(C, refs):
        assert rel(c, ref) < 2e-6
    p.close()


def test_group_beside_its_operands_is_fused():
    A, B = [mat(500, 256, i) for i in range(60)], mat(256, 256, 99)
    C = torch.empty((60 * 500, 256), device="cuda")
    p = ug.GroupedPlan([dict(ta="N", tb="N", M=500, N=256, K=256, alpha=1.0, beta=0.0, A=a, lda=256,
                             B=B, ldb=256, C=C[500 * i:], ldc=256) for i, a in enumerate(A)])
    assert p.config["fused"] == 1
    p.run()
    p.check()
    assert rel(C, torch.cat([a.double() @ B.double() for a in A])) < 2e-6
    p.close()


@pytest.mark.parametrize("M,K", [(60000, 128), (60000, 100), (300, 300), (2000, 260)])
def test_product_and_gradient_into_an_operand(M, K):
    A, B = mat(M, K, 1), mat(K, K, 2)
    ref = A.double() @ B.double()
    X = A.clone()
    ug.gemm(X, B, X, precision="bf16x6")
    assert rel(X, ref) < 2e-6
    W, d = B.t().contiguous(), A.clone()  # d: the gradient of Y in Y = X W, then of X
    ug.sgemm_backward("N", "N", M, K, K, 1.0, 0, K, W, K, d, K, 0.0, d, K, 0.0, None, K,
                      precision="bf16x6")
    assert rel(d, ref) < 2e-6
