"""Tile choices and epilogues of the single-GEMM kernels at the sizes where
they change: SIMT outputs of wide and narrow tiles mixed, split-form outputs
whose rows of C are unaligned and updated (beta != 0), against the FP64 oracle.

Normwise bound: a depth-K FP32 accumulation is within about sqrt(K) 2^-24 of
FP64 (5e-7 at K = 70); 2e-6 is the suite's bound for both forms."""
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


def check(ta, tb, M, N, K, prec, beta=0.5, pad=0):
    g = torch.Generator(device="cuda").manual_seed(M + 7 * N + 13 * K)
    mat = lambda r, c: torch.rand((r, c), device="cuda", generator=g) * 2 - 1  # noqa: E731
    A = mat(M, K) if ta == "N" else mat(K, M)
    B = mat(K, N) if tb == "N" else mat(N, K)
    buf = mat(M, N + pad)
    C = buf[:, :N]
    ref = ug.ref64(ta, tb, A, B, C.contiguous(), 1.5, beta)
    rest = buf[:, N:].clone()
    ug.gemm(A, B, C, ta=ta, tb=tb, alpha=1.5, beta=beta, precision=prec)
    torch.cuda.synchronize()
    assert float(torch.linalg.norm(C.double() - ref) / torch.linalg.norm(ref)) < 2e-6
    assert torch.equal(buf[:, N:], rest)


@pytest.mark.parametrize("ta,tb", ["NN", "NT", "TN", "TT"])
@pytest.mark.parametrize("M,N,K", [(2500, 2300, 70),    # 180 wide tiles: 152, then 28 as 56 narrow
                                   (20000, 129, 33),    # one and a bit narrow columns
                                   (2049, 2561, 40),    # last wide tile row and column nearly empty
                                   (19457, 300, 32)])   # 153 x 2 wide tiles: two left over
def test_simt_wide_and_narrow_tiles(ta, tb, M, N, K):
    check(ta, tb, M, N, K, "simt", pad=3)


@pytest.mark.parametrize("prec", ["bf16x6", "fp16x3", "tf32x3"])
@pytest.mark.parametrize("M,N,K,pad", [(257, 513, 96, 0), (129, 300, 33, 1), (300, 131, 64, 2),
                                       (2049, 4097, 64, 0)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_split_epilogue_unaligned_rows(prec, M, N, K, pad, beta):
    check("T", "N", M, N, K, prec, beta, pad)


@pytest.mark.parametrize("ta,tb", ["NN", "NT", "TN", "TT"])
@pytest.mark.parametrize("M,N,K", [(100, 6000, 500), (6000, 100, 516), (128, 25088, 96),
                                   (64, 64, 8192), (1, 4096, 300), (512, 512, 512), (896, 900, 1100)])
@pytest.mark.parametrize("off", [0, 1])
def test_split_routes(ta, tb, M, N, K, off):
    """Outputs with a short side or few tiles: operands that TMA can copy are split
    inside the GEMM kernel or cut into slices and narrow tiles, others (a base one
    float off a 16-byte boundary) beforehand; C updated, bias and LeakyReLU fused."""
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + 7 * K)

    def mat(r, c):
        ld = (c + 3) // 4 * 4
        buf = torch.rand((r * ld + 4,), device="cuda", generator=g) * 2 - 1
        return buf[off:off + r * ld].view(r, ld)[:, :c]

    A = mat(M, K) if ta == "N" else mat(K, M)
    B = mat(K, N) if tb == "N" else mat(N, K)
    C = mat(M, N)
    bias = torch.randn((M,), device="cuda", generator=g)
    ref = ug.ref64(ta, tb, A, B, C.contiguous(), 1.5, 0.5) + bias.double()[:, None]
    ref = torch.where(ref > 0, ref, 0.1 * ref)
    ug.gemm_ex(A, B, C, bias=bias, act=1, slope=0.1, ta=ta, tb=tb, alpha=1.5, beta=0.5,
               precision="bf16x6")
    torch.cuda.synchronize()
    assert float(torch.linalg.norm(C.double() - ref) / torch.linalg.norm(ref)) < 2e-6


# values in [1, 2) have scale exponent 14: 63 and 64 are reached at 2^-49 and
# 2^-50, -63 and -64 at 2^77 and 2^78
@pytest.mark.parametrize("a_exp,b_exp", [(77, 0), (78, 0), (0, 77), (0, 78), (77, -49), (78, -50),
                                         (-49, 0), (-50, 0), (0, -49), (0, -50), (-49, -49)])
def test_fp16x3_scale_limits(a_exp, b_exp):
    """A row of A (a column of B) times 2^e has its scale exponent moved by e and the
    same pieces, so C's row (column) is the plain result times 2^e to the bit, on
    both sides of the exponents (+-63) up to which one product undoes both scales."""
    M, N, K = 200, 330, 96
    g = torch.Generator(device="cuda").manual_seed(5)
    A = torch.rand((M, K), device="cuda", generator=g) + 0.5
    B = torch.rand((K, N), device="cuda", generator=g) + 0.5
    A[:, 0], B[0] = 1.75, 1.75
    plain = ug.gemm(A, B, torch.empty((M, N), device="cuda"), precision="fp16x3").clone()
    A2, B2 = A.clone(), B.clone()
    A2[5] *= 2.0 ** a_exp
    B2[:, 7] *= 2.0 ** b_exp
    out = ug.gemm(A2, B2, torch.empty((M, N), device="cuda"), precision="fp16x3")
    want = plain.clone()
    want[5] *= 2.0 ** a_exp
    want[:, 7] *= 2.0 ** b_exp
    assert torch.equal(out, want)


@pytest.mark.parametrize("M,N,K", [(256, 256, 4096), (320, 1000, 2048)])
def test_arena_for_whole_tiles_alone(M, N, K):
    """k slices need partial tiles beside the pieces; an arena that only holds the
    pieces is still enough, for whole tiles."""
    import numpy as np
    pieces = 6 * (M + N) * K
    assert ug.workspace_bytes("N", "N", M, N, K, K, N, "bf16x6") > pieces + 4096
    rng = np.random.default_rng(1)
    A, B = rng.random((M, K), np.float32) - 0.5, rng.random((K, N), np.float32) - 0.5
    C = np.zeros((M, N), np.float32)
    ug.sgemm_cuda_init(size=4 * (M * K + K * N + M * N) + pieces + 4096)
    try:
        ug.set_precision("bf16x6")
        ug.sgemm_cuda("N", "N", M, N, K, 1.0, A, B, 0.0, C)
    finally:
        ug.set_precision("auto")
        ug.sgemm_cuda_finish()
    ref = A.astype(np.float64) @ B.astype(np.float64)
    assert np.linalg.norm(C - ref) / np.linalg.norm(ref) < 2e-6


@pytest.mark.parametrize("ta,tb", ["NN", "NT", "TN", "TT"])
@pytest.mark.parametrize("M,N,K", [(2500, 2300, 270),   # the sizes above, deep enough for wide tiles
                                   (20000, 129, 257), (2049, 2561, 300), (19457, 300, 260),
                                   (128, 25088, 290),   # one wave of 128 x 192
                                   (6000, 6000, 33), (1025, 4097, 31), (4096, 4096, 8)])  # narrow ones
def test_simt_tiles_by_depth(ta, tb, M, N, K):
    check(ta, tb, M, N, K, "simt", pad=3)


def simt_us(ta, tb, M, N, K):
    A = torch.rand((M, K) if ta == "N" else (K, M), device="cuda")
    B = torch.rand((K, N) if tb == "N" else (N, K), device="cuda")
    C = torch.empty((M, N), device="cuda")
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    best = 1e9
    for _ in range(8):
        e[0].record()
        for _ in range(10):
            ug.gemm(A, B, C, ta=ta, tb=tb, precision="simt")
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]))
    return best * 100


def test_simt_shallow_time():
    """A product of one k stage is bound by its stores: it takes as long in every layout
    (in wide tiles, which NT has none of, 1.26 times as long)."""
    assert simt_us("N", "N", 6000, 6000, 32) < 1.12 * simt_us("N", "T", 6000, 6000, 32)
