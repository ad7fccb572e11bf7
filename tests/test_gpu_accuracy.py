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
