"""The error words of the device-pointer calls beside captures, replays and other
streams.  Codes are planted with a host copy (nothing faults or waits): a kernel
that finds one in its word gives up its waits and leaves its output unfinished."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
import ugemm_gb300 as ug  # noqa: E402

N = 16


@pytest.fixture(scope="module", autouse=True)
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ug.build()
    ug.load()


class Calls:
    """Many small calls, each with an output of its own, on streams in turn."""

    def __init__(self, n, *streams):
        g = torch.Generator(device="cuda").manual_seed(2)
        self.A = torch.rand((N, 64), device="cuda", generator=g)
        self.B = torch.rand((64, N), device="cuda", generator=g)
        self.C = torch.full((n, N, N), float("nan"), device="cuda")
        self.streams = streams
        torch.cuda.synchronize()

    def run(self):
        for i in range(len(self.C)):
            ug.sgemm_dev("N", "N", N, N, 64, 1.0, self.A, 64, self.B, N, 0.0, self.C[i], N,
                         precision="simt", stream=self.streams[i % len(self.streams)])

    def check(self):
        torch.cuda.synchronize()
        ref = self.A.double() @ self.B.double()
        assert float((self.C.double() - ref).abs().max()) < 1e-5   # 64 products below 1


def plant(code):
    assert ug.load().ugemm_debug_set_error_word(0, code) == ug.OK


def reported(code):
    with pytest.raises(ug.UgemmError) as err:
        ug.check()
    assert err.value.status == ug.ERR_TIMEOUT and f"code {code}" in str(err.value)
    ug.check()  # once


def test_words_come_round_without_their_codes():
    ug.check()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    calls = Calls(9001, one, two)
    ug.sgemm_dev("N", "N", N, N, 64, 1.0, calls.A, 64, calls.B, N, 0.0, calls.C[0], N,
                 precision="simt", stream=one)
    torch.cuda.synchronize()
    plant(3)
    calls.run()
    calls.check()
    reported(3)


def test_more_streams_than_rings():
    calls = Calls(200, *[torch.cuda.ExternalStream(s.cuda_stream) for s in
                         (torch.cuda.Stream(priority=p) for p in (0, -1) * 50)])
    calls.run()
    calls.check()
    ug.check()


def test_calls_beside_a_capture_on_another_stream():
    """Eager calls make nothing that a global-mode capture forbids."""
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    calls, inside = Calls(5000, two), Calls(1, one)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=one):
        inside.run()
        calls.run()
    calls.check()
    g.replay()
    inside.check()
    ug.check()


def test_captured_calls_keep_their_word():
    M, K = 1100, 1500
    A, B = torch.rand((M, K), device="cuda"), torch.rand((K, M), device="cuda")
    ref = ug.ref64("N", "N", A, B)
    C = ug.gemm(A, B, precision="bf16x6")   # the workspace it needs
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=one):
        ug.gemm(A, B, C, precision="bf16x6", stream=one)
    plant(4)                                # as a replay's kernels would leave it
    calls = Calls(9001, one, two)
    calls.run()
    calls.check()                           # no eager call was given that word
    C.fill_(float("nan"))
    g.replay()                              # nor does the replay find its code
    torch.cuda.synchronize()
    assert float(torch.linalg.norm(C.double() - ref) / torch.linalg.norm(ref)) < 2e-6
    reported(4)
    plant(5)                                # (the last call is an eager one of `two`)
    g.replay()
    torch.cuda.synchronize()
    assert float(torch.linalg.norm(C.double() - ref) / torch.linalg.norm(ref)) < 2e-6
    reported(5)
