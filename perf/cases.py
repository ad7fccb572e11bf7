"""The work that a user of ugemm_gb300 has it do, as cases that can be timed.

Sizes are the benchmark's and the tests' own (the seeded 256-problem group, the
12-layer convolution stack, 8192^3, the ragged 4095 x 4097 x 1023, the
rectangular adjoint 2048 x 8192 x 1024), and between and around them generic
ones.  ``listed`` names twelve; ``draw`` gives more of the same ranges.  A case
is run through the public entry points of the package with everything resident
that a program would keep (plans, stacks, the compat arena), on inputs made
from a seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import ugemm_gb300 as ug
from ugemm_gb300 import workloads

DEV = "cuda"


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def _stack_text(layers) -> str:
    """Layers (cin, cout, h, w, stride[, ksize, pad]) as one text value."""
    return ";".join(",".join(str(int(v)) for v in l) for l in layers)


def _stack_layers(text: str):
    return [tuple(int(v) for v in l.split(",")) for l in text.split(";")]


def listed():
    return [
        # the smallest call: a dense layer of a small model; launches and latency count
        dict(name="gemm_small", kind="gemm", ta="N", tb="T", M=64, N=48, K=96, alpha=1.0,
             beta=0.0, prec="auto", span=0),
        # an ordinary square product with the default form
        dict(name="gemm_1024", kind="gemm", ta="N", tb="N", M=1024, N=1024, K=1024, alpha=1.0,
             beta=0.0, prec="auto", span=0),
        # odd and ragged sizes, a transposed operand, C updated; values over many binades
        dict(name="gemm_ragged", kind="gemm", ta="T", tb="N", M=4095, N=4097, K=1023, alpha=1.5,
             beta=0.5, prec="auto", span=8),
        # the largest product, in the fastest split form
        dict(name="gemm_8192_fp16x3", kind="gemm", ta="N", tb="N", M=8192, N=8192, K=8192,
             alpha=1.5, beta=0.5, prec="fp16x3", span=0),
        # the plain FP32 form: every product and sum in FP32 on the CUDA cores
        dict(name="gemm_4096_simt", kind="gemm", ta="N", tb="N", M=4096, N=4096, K=4096,
             alpha=1.0, beta=0.0, prec="simt", span=0),
        # a convolution layer's forward product with its bias and LeakyReLU fused
        dict(name="layer_bias_leaky", kind="layer", M=128, N=25088, K=1152, prec="auto"),
        # the adjoint of a rectangular product: dA and dB
        dict(name="backward_rect", kind="backward", ta="N", tb="N", M=2048, N=8192, K=1024,
             prec="auto"),
        # 256 uneven products kept as one plan and replayed
        dict(name="grouped_256", kind="grouped", count=256, seed=workloads.GROUPED_SEED, lo=32,
             hi=1024, align=4, prec="bf16x6", graph=True),
        # a training step of the 12-layer convolution stack: forward, dX and dW
        dict(name="conv_train", kind="conv", layers=_stack_text(workloads.conv_layers()), batch=32,
             what=3, leaky=-1.0, prec="bf16x6", graph=True),
        # the same network looking at one image, with its activations
        dict(name="conv_infer", kind="conv", layers=_stack_text(workloads.conv_layers()), batch=1,
             what=1, leaky=0.1, prec="bf16x6", graph=True),
        # the reference's own call: host pointers in plain memory, device arena kept
        dict(name="host_2048", kind="host", ta="N", tb="N", M=2048, N=2048, K=2048, alpha=1.0,
             beta=0.0),
        # a dense layer applied to one vector
        dict(name="gemv_8192", kind="gemv", trans="T", M=8192, N=8192, incx=1, incy=1, alpha=1.0,
             beta=0.0),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5 and v >= 64:  # half of the larger sizes are multiples of 32
        v = v // 32 * 32
    return max(lo, min(hi, v))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "gemm", "layer", "backward", "grouped", "conv", "host",
                       "gemv"])
    t = lambda: rng.choice("NT")  # noqa: E731
    if kind == "gemm":
        prec = rng.choice(["auto", "auto", "simt", "bf16x6", "fp16x3"])
        hi = 4096 if prec == "simt" else 8192
        beta = rng.choice([0.0, 0.0, 0.5])
        return dict(kind=kind, ta=t(), tb=t(), M=_log_int(rng, 32, hi), N=_log_int(rng, 32, hi),
                    K=_log_int(rng, 32, hi), alpha=rng.choice([1.0, 1.5]), beta=beta, prec=prec,
                    span=rng.choice([0, 8]))
    if kind == "layer":
        return dict(kind=kind, M=_log_int(rng, 64, 512), N=_log_int(rng, 1568, 100352),
                    K=_log_int(rng, 64, 2304), prec=rng.choice(["auto", "bf16x6"]))
    if kind == "backward":
        return dict(kind=kind, ta=t(), tb=t(), M=_log_int(rng, 64, 4096), N=_log_int(rng, 64, 8192),
                    K=_log_int(rng, 64, 4096), prec=rng.choice(["auto", "auto", "bf16x6", "fp16x3"]))
    if kind == "grouped":
        return dict(kind=kind, count=rng.randint(8, 256), seed=rng.randrange(1 << 20),
                    lo=rng.choice([16, 32, 64]), hi=rng.choice([512, 1024]),
                    align=rng.choice([1, 4, 4]), prec=rng.choice(["bf16x6", "bf16x6", "simt"]),
                    graph=rng.choice([True, False]))
    if kind == "conv":
        batch = _log_int(rng, 1, 32)
        size = rng.choice([7, 13, 14, 28, 32, 56])
        cin = rng.choice([3, 16, 32, 64, 96, 128, 256])
        cout = rng.choice([32, 64, 128, 200, 256])
        layers = []
        for i in range(rng.randint(1, 3)):
            k = rng.choice([3, 3, 3, 1])
            stride = rng.choice([1, 1, 2]) if size > 4 else 1
            pad = k // 2
            layers.append((cin, cout, size, size, stride, k, pad))
            size = (size + 2 * pad - k) // stride + 1
            cin = cout
        return dict(kind=kind, layers=_stack_text(layers), batch=batch, what=rng.choice([1, 3]),
                    leaky=rng.choice([-1.0, 0.1]), prec="bf16x6", graph=rng.choice([True, True, False]))
    if kind == "host":
        return dict(kind=kind, ta=t(), tb=t(), M=_log_int(rng, 32, 2048),
                    N=_log_int(rng, 32, 2048), K=_log_int(rng, 32, 2048), alpha=1.0,
                    beta=rng.choice([0.0, 0.5]))
    return dict(kind="gemv", trans=t(), M=_log_int(rng, 64, 8192), N=_log_int(rng, 64, 8192),
                incx=1, incy=rng.choice([1, 1, 2]), alpha=rng.choice([1.0, 1.5]),
                beta=rng.choice([0.0, 0.5]))


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(seed)


def _matrix(rows: int, cols: int, g, span: int = 0) -> torch.Tensor:
    """U[-1, 1); with span s: mantissa U[1, 2), random sign, exponents in [-s, s]."""
    if span == 0:
        return torch.rand((rows, cols), device=DEV, generator=g) * 2 - 1
    m = torch.rand((rows, cols), device=DEV, generator=g) + 1
    s = torch.randint(0, 2, (rows, cols), device=DEV, generator=g) * 2 - 1
    e = torch.randint(-span, span + 1, (rows, cols), device=DEV, generator=g)
    return torch.ldexp(m * s, e)


def _stored(t: str, rows: int, cols: int):
    return (rows, cols) if t == "N" else (cols, rows)


def _gemm_inputs(c, seed):
    g = _gen(seed)
    A = _matrix(*_stored(c["ta"], c["M"], c["K"]), g, c["span"])
    B = _matrix(*_stored(c["tb"], c["K"], c["N"]), g, c["span"])
    C = _matrix(c["M"], c["N"], g) if c["beta"] else torch.zeros((c["M"], c["N"]), device=DEV)
    return A, B, C


def _layer_inputs(c, seed):
    g = _gen(seed)
    W = torch.randn((c["M"], c["K"]), device=DEV, generator=g) * (2.0 / c["K"]) ** 0.5
    X = torch.rand((c["K"], c["N"]), device=DEV, generator=g)
    bias = torch.randn((c["M"],), device=DEV, generator=g) * 0.1
    return W, X, bias


def _backward_inputs(c, seed):
    g = _gen(seed)
    A = _matrix(*_stored(c["ta"], c["M"], c["K"]), g)
    B = _matrix(*_stored(c["tb"], c["K"], c["N"]), g)
    dC = torch.randn((c["M"], c["N"]), device=DEV, generator=g)
    return A, B, dC


def _round_up(x: int, a: int) -> int:
    return -(-x // a) * a


def _grouped_specs(c, seed):
    """The group's problems on flat buffers (rows padded to `align` floats, matrices on
    16-byte boundaries when align is 4), C's buffer returned whole."""
    shapes = workloads.grouped_shapes(c["count"], c["seed"], c["lo"], c["hi"])
    al = c["align"]
    rows, ab, cc = [], 0, 0
    for ta, tb, M, N, K in shapes:
        (ar, ac), (br, bc) = _stored(ta, M, K), _stored(tb, K, N)
        lda, ldb, ldc = _round_up(ac, al), _round_up(bc, al), _round_up(N, al)
        rows.append((ta, tb, M, N, K, ab, lda, ab + ar * lda, ldb, cc, ldc))
        ab += ar * lda + br * ldb
        cc += M * ldc
    flat = torch.rand((ab,), device=DEV, generator=_gen(seed)) * 2 - 1
    out = torch.zeros((cc,), device=DEV)
    return rows, flat, out


def _conv_inputs(c, seed):
    """x0: U[0, 1) activations; He-normal weights; small biases."""
    g = _gen(seed)
    layers = _stack_layers(c["layers"])
    cin, _, h, w = layers[0][:4]
    x = torch.rand((cin, c["batch"] * h * w), device=DEV, generator=g)
    ws, bs = [], []
    for l in layers:
        k = l[5] if len(l) > 5 else 3
        kd = l[0] * k * k
        ws.append(torch.randn((l[1], kd), device=DEV, generator=g) * (2.0 / kd) ** 0.5)
        bs.append(torch.randn((l[1],), device=DEV, generator=g) * 0.1)
    return layers, x, ws, bs


def _conv_geometry(layers):
    """Per layer (cin, cout, h, w, stride, k, pad, ho, wo)."""
    out = []
    for l in layers:
        cin, cout, h, w, s = l[:5]
        k, p = (l[5], l[6]) if len(l) > 5 else (3, 1)
        out.append((cin, cout, h, w, s, k, p, (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1))
    return out


def _host_inputs(c, seed):
    rng = np.random.default_rng(seed)
    mat = lambda r, k: rng.random((r, k), dtype=np.float32) * 2 - 1  # noqa: E731
    A = mat(*_stored(c["ta"], c["M"], c["K"]))
    B = mat(*_stored(c["tb"], c["K"], c["N"]))
    C = mat(c["M"], c["N"]) if c["beta"] else np.zeros((c["M"], c["N"]), np.float32)
    return A, B, C


def _gemv_inputs(c, seed):
    """A column-major, stored as the torch matrix of its columns: M x N for 'N', N x M for 'T'."""
    g = _gen(seed)
    cols, lda = (c["N"], c["M"]) if c["trans"] == "N" else (c["M"], c["N"])
    A = _matrix(cols, lda, g)
    x = _matrix(1, c["N"] * c["incx"], g).reshape(-1)
    y = _matrix(1, c["M"] * c["incy"], g).reshape(-1)
    return A, x, y


_ARENA = []


def _arena():
    """The process's one compat context, as the reference's test sets it up: ten times the
    matrices of the largest call in these ranges."""
    if not _ARENA:
        ug.sgemm_cuda_init(0, torch.cuda.current_device(), 3 * 2048 * 2048 * 10 * 4)
        _ARENA.append(True)


def prepare(case, seed):
    k = case["kind"]
    if k == "gemm":
        return (case, *_gemm_inputs(case, seed))
    if k == "layer":
        W, X, bias = _layer_inputs(case, seed)
        return case, W, X, bias, torch.empty((case["M"], case["N"]), device=DEV)
    if k == "backward":
        A, B, dC = _backward_inputs(case, seed)
        return case, A, B, dC, torch.empty_like(A), torch.empty_like(B)
    if k == "grouped":
        rows, flat, out = _grouped_specs(case, seed)
        base, obase = flat.data_ptr(), out.data_ptr()
        specs = [dict(ta=ta, tb=tb, M=M, N=N, K=K, alpha=1.0, beta=0.0, A=base + 4 * a, lda=lda,
                      B=base + 4 * b, ldb=ldb, C=obase + 4 * c, ldc=ldc)
                 for ta, tb, M, N, K, a, lda, b, ldb, c, ldc in rows]
        return case, ug.GroupedPlan(specs, precision=case["prec"], graph=case["graph"]), flat, out
    if k == "conv":
        layers, x, ws, bs = _conv_inputs(case, seed)
        leaky = None if case["leaky"] < 0 else case["leaky"]
        stack = ug.ConvStack(layers, case["batch"], precision=case["prec"], graph=case["graph"],
                             leaky=leaky)
        stack.tensor(0, "x", x.shape).copy_(x)
        for l in range(len(layers)):
            stack.tensor(l, "w", ws[l].shape).copy_(ws[l])
            stack.tensor(l, "bias", bs[l].shape).copy_(bs[l])
        outs = {}
        for l, (cin, cout, h, w, s, kk, p, ho, wo) in enumerate(_conv_geometry(layers)):
            n = case["batch"] * ho * wo
            if case["what"] & ug.CONV_BACKWARD:
                outs[f"dw{l}"] = stack.tensor(l, "dw", (cout, cin * kk * kk))
                if leaky is not None:
                    outs[f"dbias{l}"] = stack.tensor(l, "dbias", (cout,))
                if l == 0:
                    outs["dx0"] = stack.tensor(0, "dx", (cin, case["batch"] * h * w))
                if l + 1 < len(layers):
                    outs[f"y{l}"] = stack.tensor(l, "y", (cout, n))
            else:
                outs[f"y{l}"] = stack.tensor(l, "y", (cout, n))
        for t in outs.values():  # views of the stack's own memory: it lives as long as they do
            t.owner = stack
        return case, stack, outs
    if k == "host":
        _arena()
        return (case, *_host_inputs(case, seed))
    return (case, *_gemv_inputs(case, seed))


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(state):
    case = state[0]
    k = case["kind"]
    if k == "gemm":
        _, A, B, C = state
        return ug.gemm(A, B, C, ta=case["ta"], tb=case["tb"], alpha=case["alpha"],
                       beta=case["beta"], precision=case["prec"])
    if k == "layer":
        _, W, X, bias, Y = state
        return ug.gemm_ex(W, X, Y, bias=bias, act=1, slope=0.1, precision=case["prec"])
    if k == "backward":
        _, A, B, dC, dA, dB = state
        M, N, K = case["M"], case["N"], case["K"]
        ug.sgemm_backward(case["ta"], case["tb"], M, N, K, 1.0, A, A.stride(0), B, B.stride(0), dC,
                          N, 0.0, dA, dA.stride(0), 0.0, dB, dB.stride(0), precision=case["prec"])
        return dA, dB
    if k == "grouped":
        state[1].run()
        return state[3]
    if k == "conv":
        state[1].run(case["what"])
        return state[2]
    if k == "host":
        _, A, B, C = state
        ug.sgemm_cuda(case["ta"], case["tb"], case["M"], case["N"], case["K"], case["alpha"], A, B,
                      case["beta"], C)
        return C
    _, A, x, y = state
    ug.sgemv(case["trans"], case["M"], case["N"], case["alpha"], A, A.stride(0), x, case["incx"],
             case["beta"], y, case["incy"])
    return y


# --------------------------------------------------------------------------
# what a pass cannot do without, and what it should give
# --------------------------------------------------------------------------
def work(case):
    k = case["kind"]
    if k in ("gemm", "host"):
        M, N, K = case["M"], case["N"], case["K"]
        c = M * N * (2 if case["beta"] else 1)
        return {"bytes": 4 * (M * K + K * N + c), "flops": 2.0 * M * N * K}
    if k == "layer":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 4 * (M * K + K * N + M * N + M), "flops": 2.0 * M * N * K}
    if k == "backward":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 4 * (2 * M * K + 2 * K * N + M * N), "flops": 4.0 * M * N * K}
    if k == "grouped":
        b = f = 0
        for _, _, M, N, K in workloads.grouped_shapes(case["count"], case["seed"], case["lo"],
                                                      case["hi"]):
            b += 4 * (M * K + K * N + M * N)
            f += 2.0 * M * N * K
        return {"bytes": b, "flops": f}
    if k == "conv":
        b = f = 0
        for cin, cout, h, w, s, kk, p, ho, wo in _conv_geometry(_stack_layers(case["layers"])):
            x, y, wt = cin * case["batch"] * h * w, cout * case["batch"] * ho * wo, cout * cin * kk * kk
            one = 2.0 * y * cin * kk * kk
            b += 4 * (x + wt + y)
            f += one
            if case["what"] & ug.CONV_BACKWARD:  # dY, W and X in, dX and dW out
                b += 4 * (y + wt + x + x + wt)
                f += 2 * one
        return {"bytes": b, "flops": f}
    M, N = case["M"], case["N"]
    return {"bytes": 4 * (M * N + N + M * (2 if case["beta"] else 1)), "flops": 2.0 * M * N}


def _op(X, t):
    return X.double() if t == "N" else X.double().T


def _exact_conv(case, seed):
    layers, x, ws, bs = _conv_inputs(case, seed)
    geo = _conv_geometry(layers)
    B, leaky = case["batch"], case["leaky"]
    cin, _, h, w = geo[0][:4]
    a = x.double().reshape(cin, B, h, w).permute(1, 0, 2, 3).contiguous()
    saved, outs = [], {}
    for l, (ci, co, hh, ww, s, k, p, ho, wo) in enumerate(geo):
        cols = torch.nn.functional.unfold(a, k, padding=p, stride=s)      # B, ci k k, ho wo
        cols = cols.permute(1, 0, 2).reshape(ci * k * k, B * ho * wo)
        y = ws[l].double() @ cols
        if leaky >= 0:
            y = torch.nn.functional.leaky_relu(y + bs[l].double()[:, None], leaky)
        saved.append(cols if case["what"] & ug.CONV_BACKWARD else None)
        outs[f"y{l}"] = y
        a = y.reshape(co, B, ho, wo).permute(1, 0, 2, 3).contiguous()
    if not case["what"] & ug.CONV_BACKWARD:
        return outs
    d = outs.pop(f"y{len(geo) - 1}")   # the last output is its own incoming gradient
    top = d
    for l in range(len(geo) - 1, -1, -1):
        ci, co, hh, ww, s, k, p, ho, wo = geo[l]
        if leaky >= 0:
            y = top if l == len(geo) - 1 else outs[f"y{l}"]
            d = torch.where(y > 0, d, d * leaky)
            outs[f"dbias{l}"] = d.sum(1)
        outs[f"dw{l}"] = d @ saved[l].T
        saved[l] = None
        dcol = (ws[l].double().T @ d).reshape(ci * k * k, B, ho * wo).permute(1, 0, 2)
        d = torch.nn.functional.fold(dcol, (hh, ww), k, padding=p, stride=s)
        d = d.permute(1, 0, 2, 3).reshape(ci, B * hh * ww)
    outs["dx0"] = d
    return outs


def exact(case, seed):
    k = case["kind"]
    if k == "gemm":
        A, B, C = _gemm_inputs(case, seed)
        return case["alpha"] * (_op(A, case["ta"]) @ _op(B, case["tb"])) + case["beta"] * C.double()
    if k == "layer":
        W, X, bias = _layer_inputs(case, seed)
        y = W.double() @ X.double() + bias.double()[:, None]
        return torch.where(y > 0, y, y * 0.1)
    if k == "backward":
        A, B, dC = _backward_inputs(case, seed)
        a, b, d = _op(A, case["ta"]), _op(B, case["tb"]), dC.double()
        dA, dB = d @ b.T, a.T @ d
        return (dA if case["ta"] == "N" else dA.T.contiguous(),
                dB if case["tb"] == "N" else dB.T.contiguous())
    if k == "grouped":
        rows, flat, out = _grouped_specs(case, seed)
        out = out.double()
        for ta, tb, M, N, K, a, lda, b, ldb, c, ldc in rows:
            (ar, ac), (br, bc) = _stored(ta, M, K), _stored(tb, K, N)
            A = flat[a:a + ar * lda].view(ar, lda)[:, :ac]
            B = flat[b:b + br * ldb].view(br, ldb)[:, :bc]
            out[c:c + M * ldc].view(M, ldc)[:, :N] = _op(A, ta) @ _op(B, tb)
        return out
    if k == "conv":
        return _exact_conv(case, seed)
    if k == "host":
        A, B, C = (torch.from_numpy(v).to(DEV) for v in _host_inputs(case, seed))
        r = case["alpha"] * (_op(A, case["ta"]) @ _op(B, case["tb"])) + case["beta"] * C.double()
        return r.cpu().numpy()
    A, x, y = _gemv_inputs(case, seed)
    A64 = A.double().T if case["trans"] == "N" else A.double()
    out = y.double().clone()
    at = torch.arange(case["M"], device=DEV) * case["incy"]
    out[at] = case["alpha"] * (A64 @ x.double()[::case["incx"]][:case["N"]]) + case["beta"] * out[at]
    return out
