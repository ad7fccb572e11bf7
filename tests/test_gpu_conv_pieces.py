"""Convolution layers whose GEMMs read their im2col operands from NHWC pieces
(three-piece forms): channel counts that pad their 32- and 64-channel blocks,
kernel sizes 1, 3 and 5, strides, pads below the "same" one, images narrower
than a tile's pixels, a few channels (gathered instead), against FP64.

Bound: FP32-grade accumulation of depth K, max(2e-6, 2.5e-8 sqrt(K)), as for
the 12-layer stack; the deepest here is 9 x 256."""
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


def rel(a, b):
    return float(torch.linalg.norm(a.double() - b) / torch.linalg.norm(b))


LAYERS = [  # (cin, cout, h, w, stride, ksize, pad), batch
    ((64, 64, 8, 8, 1, 3, 1), 4), ((32, 64, 9, 7, 1, 3, 1), 2), ((64, 128, 9, 7, 2, 3, 1), 3),
    ((96, 200, 14, 14, 1, 3, 1), 5), ((64, 32, 13, 13, 1, 1, 0), 2), ((48, 40, 10, 11, 1, 5, 2), 3),
    ((128, 256, 7, 7, 1, 3, 1), 1), ((256, 96, 5, 3, 1, 3, 1), 7), ((128, 128, 12, 12, 1, 3, 0), 2),
    ((64, 72, 31, 1, 2, 3, 1), 2), ((3, 64, 12, 12, 1, 3, 1), 2)]


@pytest.mark.parametrize("prec", ["bf16x6", "bf16x9"])
@pytest.mark.parametrize("layer,batch", LAYERS)
@pytest.mark.parametrize("separate", [False, True])  # forward and backward as two runs
def test_layer_against_fp64(prec, layer, batch, separate):
    cin, cout, h, w, s, k, p = layer
    ho, wo = (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    stack = ug.ConvStack([layer], batch, precision=prec, graph=not separate)
    x = stack.tensor(0, "x", (cin, batch, h, w))
    x.copy_(torch.rand(x.shape, device="cuda", generator=g) - 0.3)
    wt = stack.tensor(0, "w", (cout, cin, k, k))
    wt.copy_(torch.randn(wt.shape, device="cuda", generator=g))
    if separate:
        stack.run(ug.CONV_FORWARD)
        stack.run(ug.CONV_BACKWARD)
    else:
        stack.run()
    torch.cuda.synchronize()
    xd = x.double().permute(1, 0, 2, 3).contiguous().requires_grad_()
    wd = wt.double().clone().requires_grad_()
    cols = torch.nn.functional.unfold(xd, k, padding=p, stride=s)
    yd = wd.reshape(cout, -1) @ cols
    y = stack.tensor(0, "y", (cout, batch, ho * wo))
    (0.5 * (yd * yd).sum()).backward()
    tol = lambda depth: max(2e-6, 2.5e-8 * depth ** 0.5)  # noqa: E731
    assert rel(y.permute(1, 0, 2), yd.detach()) < tol(cin * k * k)
    assert rel(stack.tensor(0, "dw", wt.shape), wd.grad) < tol(batch * ho * wo)
    dx = stack.tensor(0, "dx", (cin, batch, h, w)).permute(1, 0, 2, 3)
    assert rel(dx, xd.grad) < tol(cout * k * k)
    stack.close()


# edges of the weight split's tiles (72 taps x rows, 64 / 32 / 16 channels of up
# to 72 / 144 / 256 taps): ragged rows and channels, one tap, even kernels, and
# kernels on both sides of each limit
@pytest.mark.parametrize("layer,batch", [
    ((22, 33, 9, 9, 1, 3, 1), 2), ((70, 65, 9, 9, 1, 3, 1), 1), ((64, 33, 8, 8, 2, 1, 0), 2),
    ((40, 47, 9, 9, 1, 2, 1), 1), ((72, 40, 10, 10, 1, 8, 4), 1), ((44, 70, 10, 10, 1, 9, 4), 1),
    ((64, 44, 13, 13, 1, 12, 6), 1), ((44, 23, 14, 14, 1, 13, 6), 1),
    ((64, 64, 17, 17, 1, 16, 8), 1)])
def test_weight_split_tiles(layer, batch):
    test_layer_against_fp64("bf16x6", layer, batch, False)


def test_backward_alone_reads_the_inputs_it_is_given():
    """A backward run splits X itself: writing X between the two runs counts."""
    layer, batch = (64, 64, 8, 8, 1, 3, 1), 2
    stack = ug.ConvStack([layer], batch, precision="bf16x6", graph=True)
    g = torch.Generator(device="cuda").manual_seed(1)
    x, wt = stack.tensor(0, "x", (64, batch * 64)), stack.tensor(0, "w", (64, 576))
    x.copy_(torch.rand(x.shape, device="cuda", generator=g))
    wt.copy_(torch.randn(wt.shape, device="cuda", generator=g))
    stack.run(ug.CONV_FORWARD)
    x.mul_(2)
    stack.run(ug.CONV_BACKWARD)
    torch.cuda.synchronize()
    two = stack.tensor(0, "dw", (64, 576)).clone()
    x.mul_(0.5)
    stack.run(ug.CONV_BACKWARD)
    torch.cuda.synchronize()
    assert torch.equal(two, 2 * stack.tensor(0, "dw", (64, 576)))
    stack.close()


def test_small_input_is_split_with_the_weights():
    """One launch splits the weights of all layers and a small first input."""
    stack = ug.ConvStack([(96, 96, 14, 14, 1, 1, 0)], 1, precision="bf16x6", graph=False)
    stack.run(ug.CONV_FORWARD)
    ug.profile_enable(True)
    ug.profile_collect()
    try:
        stack.run(ug.CONV_FORWARD)
        assert ug.profile_collect()["split_prepass"][1] == 1
    finally:
        ug.profile_enable(False)
        stack.close()
