"""Norm with a pass-through output and dropout with a residual: the same values and masks as the separate calls."""
import pytest
import torch

from merak_b200.ops.elementwise import dropout, dropout_add
from merak_b200.ops.norm import fused_norm, norm_fork
from merak_b200.ops.rng import dropout_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,H", [(1, 8), (5, 768), (33, 1024), (7, 1600), (3, 8192)])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("use", ["both", "norm", "pass"])
def test_norm_fork(M, H, rms, use):
    torch.manual_seed(M + H)
    x0 = torch.randn(M, H, device="cuda").bfloat16()
    w0 = torch.randn(H, device="cuda").bfloat16()
    b0 = None if rms else torch.randn(H, device="cuda").bfloat16()
    g, r = torch.randn_like(x0), torch.randn_like(x0)
    grads, outs = [], []
    for fork in (True, False):
        x, w = x0.clone().requires_grad_(True), w0.clone().requires_grad_(True)
        b = None if b0 is None else b0.clone().requires_grad_(True)
        y, z = norm_fork(x, w, b, 1e-5, rms) if fork else (fused_norm(x, w, b, None, 1e-5, rms)[0], x)
        loss = 0.0
        if use != "pass":
            loss = loss + (y.float() * g.float()).sum()
        if use != "norm":
            loss = loss + (z.float() * r.float()).sum()
        loss.backward()
        outs.append((y.detach(), z.detach()))
        grads.append([x.grad] + ([w.grad] if use != "pass" else []))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    for a, b in zip(*grads):       # one rounding to bf16 instead of two
        assert (a.float() - b.float()).norm() <= 2.0 ** -7 * b.float().norm()


@pytest.mark.parametrize("shape", [(8,), (3, 5, 768), (2, 1001, 8), (1, 7)])
@pytest.mark.parametrize("p", [0.0, 0.1, 0.9])
@pytest.mark.parametrize("training", [True, False])
def test_dropout_add(shape, p, training):
    torch.manual_seed(1)
    x0, r0 = torch.randn(shape, device="cuda").bfloat16(), torch.randn(shape, device="cuda").bfloat16()
    g = torch.randn(shape, device="cuda").bfloat16()
    st, call = dropout_state(), dropout_state().get_call_id()
    res = []
    for fused in (True, False):
        st.set_call_id(call)
        x, r = x0.clone().requires_grad_(True), r0.clone().requires_grad_(True)
        y = dropout_add(x, r, p, training) if fused else dropout(x, p, training) + r
        y.backward(g)
        res.append((y.detach(), x.grad, r.grad, st.get_call_id()))
    assert res[0][3] == res[1][3]
    assert torch.equal(res[0][1], res[1][1]) and torch.equal(res[0][2], res[1][2])
    # the sum is rounded once instead of twice
    assert (res[0][0].float() - res[1][0].float()).norm() <= 2.0 ** -8 * res[1][0].float().norm()
