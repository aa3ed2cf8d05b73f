"""Gradients of one and two linear layers sharing their input, on operands as they are stored.

Against float64 products of the same 16-bit operands: fp32 accumulation over n terms and one rounding of the result,
so at most one unit in the last place (2^-8 in bf16, 2^-11 in fp16) of the norm.
"""

import threading

import pytest
import torch

from probjax_b200 import cache as C
from _gpu_util import dev, randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("m,k,n0,n1", [(64, 64, 64, 64), (65, 576, 200, 136), (300, 520, 3072, 2048), (1000, 192, 72, 328),
                                       (40, 64, 64, 64), (130, 100, 96, 64)])  # the last two: the general path
def test_pair_against_float64(m, k, n0, n1, dtype):
    d = dev()
    x, w0, w1 = randn((m, k), dtype, 1).to(d), randn((n0, k), dtype, 2).to(d), randn((n1, k), dtype, 3).to(d)
    g0, g1 = randn((m, n0), dtype, 4).to(d), randn((m, n1), dtype, 5).to(d)
    tol = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11, torch.float32: 1e-5}[dtype]

    def check(name, got, want):
        err = float((got.double() - want).norm() / want.norm())
        assert got.shape == want.shape and err <= tol, f"{name}: {err:.2e}"

    ins = [t.clone().requires_grad_(True) for t in (x, w0, w1)]
    y0, y1 = C.linear_pair_autograd(*ins)
    check("y0", y0.detach(), x.double() @ w0.double().T)
    check("y1", y1.detach(), x.double() @ w1.double().T)
    dx, dw0, dw1 = torch.autograd.grad([y0, y1], ins, [g0, g1])
    check("dx", dx, g0.double() @ w0.double() + g1.double() @ w1.double())
    check("dw0", dw0, g0.double().T @ x.double())
    check("dw1", dw1, g1.double().T @ x.double())
    # one layer, and only some of the gradients
    x2, w2 = x.clone().requires_grad_(True), w0.clone().requires_grad_(True)
    dx, dw0 = torch.autograd.grad(C.linear_autograd(x2, w2), [x2, w2], g0)
    check("dx of one layer", dx, g0.double() @ w0.double())
    check("dw of one layer", dw0, g0.double().T @ x.double())
    w3 = w1.clone().requires_grad_(True)
    y0, y1 = C.linear_pair_autograd(x, w0, w3)
    check("dw1 alone", torch.autograd.grad(y1, w3, g1)[0], g1.double().T @ x.double())


def test_weights_elsewhere_and_of_another_rank():
    """As in ``linear``: weights are moved to the device of ``x`` (their gradients come back), other ranks are refused."""
    d = dev()
    x = randn((70, 64), torch.bfloat16, 1).to(d).requires_grad_(True)
    ws = [randn((n, 64), torch.bfloat16, n).requires_grad_(True) for n in (72, 80)]  # on the host
    gs = [randn((70, n), torch.bfloat16, 3).to(d) for n in (72, 80)]
    ons = [w.detach().to(d).requires_grad_(True) for w in ws]
    got = torch.autograd.grad(C.linear_pair_autograd(x, *ws), [x, *ws], gs)
    want = torch.autograd.grad(C.linear_pair_autograd(x, *ons), [x, *ons], gs)
    assert all(not g.is_cuda for g in got[1:]) and all(torch.equal(a.to(d), b) for a, b in zip(got, want))
    one = torch.autograd.grad(C.linear_autograd(x, ws[0]), [x, ws[0]], gs[0])
    assert torch.equal(one[1], got[1])
    with pytest.raises(ValueError, match="weight"):
        C.linear_pair_autograd(x, ons[0], ons[1].view(2, 40, 64))


def test_first_call_of_a_thread_inside_a_capture():
    """The device context is bound on a thread's first tensor-core call by a means that stream capture allows."""
    d = dev()
    x, w = randn((128, 64), torch.bfloat16, 1).to(d), randn((64, 64), torch.bfloat16, 2).to(d)
    want = C.linear(x, w)  # (the status word exists from here on)
    graph, out = torch.cuda.CUDAGraph(), []

    def capture():
        try:
            with torch.cuda.device(d), torch.cuda.graph(graph, stream=torch.cuda.Stream(d)):
                out.append(C.linear(x, w))
        except Exception as e:
            out.append(e)

    thread = threading.Thread(target=capture)
    thread.start()
    thread.join()
    assert isinstance(out[0], torch.Tensor), out
    graph.replay()
    torch.cuda.synchronize(d)
    assert torch.equal(out[0], want)
