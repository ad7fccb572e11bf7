"""Device-pointer calls captured in a workspace that holds their operands' pieces and
nothing else: no k slices, whose partial tiles would need more.  In a process of its
own, as the workspace never shrinks."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
import ugemm_gb300 as ug  # noqa: E402

SCRIPT = """
import sys, torch, ugemm_gb300 as ug
what, prec, M, N, K, planes = sys.argv[1], sys.argv[2], *map(int, sys.argv[3:])
g = torch.Generator(device="cuda").manual_seed(M + N)
A = torch.rand((M, K), device="cuda", generator=g) - 0.5
B = torch.rand((K, N), device="cuda", generator=g) - 0.5
C = torch.empty((M, N), device="cuda")
ug.sgemm_dev("N", "N", 16, 16, 16, 1.0, A, K, B, N, 0.0, C, N, precision="simt")
ug.reserve_workspace(2 * planes * (M + N) * K + 8 * (M + N) + 1024)  # rounded up to 2 MiB
Bt = B.t().contiguous()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
    if what == "gemm":
        ug.gemm(A, B, C, precision=prec)
    else:  # C as the gradient of X in Y = X W with W = B^T, A the gradient of Y
        ug.sgemm_backward("N", "N", M, K, N, 1.0, 0, N, Bt, K, A, K, 0.0, C, N, 0.0, None, K,
                          precision=prec)
graph.replay()
torch.cuda.synchronize()
ref = A.double() @ B.double()
err = float(torch.linalg.norm(C.double() - ref) / torch.linalg.norm(ref))
ug.check()
assert err < 2e-6, err
"""


@pytest.fixture(scope="module", autouse=True)
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ug.build()


@pytest.mark.parametrize("what", ["gemm", "gradient"])
@pytest.mark.parametrize("prec,planes", [("bf16x6", 3), ("fp16x3", 2)])
@pytest.mark.parametrize("M,N,K", [(1024, 1024, 8192), (512, 512, 8192)])
def test_captured_without_room_for_slices(what, prec, planes, M, N, K):
    ug.load()
    assert ug.workspace_bytes("N", "N", M, N, K, K, N, prec) > 2 * planes * (M + N) * K + (4 << 20)
    root = os.path.dirname(os.path.dirname(os.path.abspath(ug.__file__)))
    r = subprocess.run([sys.executable, "-c", SCRIPT, what, prec, str(M), str(N), str(K),
                        str(planes)], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
