"""Norm kernels whose blocks walk several rows (the next row in flight, reduction buffers in turn), row by row against
fp64 PyTorch."""
import pytest
import torch

from merak_b200.ops.elementwise import dropout
from merak_b200.ops.norm import fused_norm, norm_fork
from merak_b200.ops.rng import dropout_state

pytestmark = pytest.mark.gpu

EPS = 1e-5


def _rows(H):
    """At least four rows for every block that can be resident (2048 threads per SM, blocks of 128 or 256), and a tail
    that leaves most blocks one row short."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return 4 * sms * (16 if H <= 2048 else 8) + 7


def _norm(z, w, b, rms):
    if rms:
        return z * torch.rsqrt(z.pow(2).mean(-1, keepdim=True) + EPS) * w
    return torch.nn.functional.layer_norm(z, z.shape[-1:], w, b, EPS)


def _check_rows(got, want, tol):
    err, size = (got.double() - want).norm(dim=-1), want.norm(dim=-1)
    bad = (err > tol * size + 1e-6).nonzero().flatten()
    assert bad.numel() == 0, (bad[:8].tolist(), (err / size).max().item())


@pytest.mark.parametrize("H", [776, 1600, 2048, 2056, 4096, 8192])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("form", ["plain", "fork", "residual", "dropout"])
def test_every_row(H, rms, form):
    torch.manual_seed(H)
    M = _rows(H)
    # rows of very different size and offset: a statistic or a gradient of another row shows
    size = torch.exp(torch.randn(M, 1, device="cuda"))
    x0 = (torch.randn(M, H, device="cuda") * size + torch.randn(M, 1, device="cuda") * size).bfloat16()
    r0 = (torch.randn(M, H, device="cuda") * size).bfloat16() if form in ("residual", "dropout") else None
    w0 = torch.randn(H, device="cuda").bfloat16()
    b0 = None if rms else torch.randn(H, device="cuda").bfloat16()
    gy, gz = (torch.randn(M, H, device="cuda").bfloat16() for _ in range(2))
    p = 0.25 if form == "dropout" else 0.0
    x, w = x0.clone().requires_grad_(True), w0.clone().requires_grad_(True)
    b = None if b0 is None else b0.clone().requires_grad_(True)
    r = None if r0 is None else r0.clone().requires_grad_(True)
    mask = torch.ones(M, H, device="cuda", dtype=torch.float64)
    if p > 0:
        st, call = dropout_state(), dropout_state().get_call_id()
        mask = dropout(torch.ones(M, H, device="cuda").bfloat16(), p).ne(0).double() / (1 - p)
        st.set_call_id(call)
    y, z = norm_fork(x, w, b, EPS, rms) if form == "fork" else fused_norm(x, w, b, r, EPS, rms, p)
    torch.autograd.backward((y,) if form == "plain" else (y, z), (gy,) if form == "plain" else (gy, gz))

    want_z = x0.double() * mask + (0 if r0 is None else r0.double())
    _check_rows(z.detach(), want_z, 2.0 ** -8)                       # one rounding to bf16
    zd = z.detach().double().requires_grad_(True)                    # the kernels go on with the rounded sum
    wd = w0.double().requires_grad_(True)
    bd = None if b0 is None else b0.double().requires_grad_(True)
    yd = _norm(zd, wd, bd, rms)
    _check_rows(y.detach(), yd.detach(), 2.0 ** -8)
    torch.autograd.backward((yd,), (gy.double(),))
    dz = zd.grad + (0 if form == "plain" else gz.double())
    # one rounding of each gradient; the fp32 sums behind it are off by some 2^-20 of the row
    if r is not None:
        _check_rows(r.grad, dz, 2.0 ** -8)
    _check_rows(x.grad, dz * mask, 2.0 ** -8)
    for got, want in ((w, wd), (b, bd)):
        if got is not None:
            assert (got.grad.double() - want.grad).norm() <= 2.0 ** -8 * want.grad.norm()


@pytest.mark.parametrize("H", [100, 8200])
def test_dropout_of_widths_the_norm_kernel_does_not_take(H):
    """The mask is the dropout kernel's, drawn on the device: a captured call draws a new one at every replay."""
    st = dropout_state()
    x, r = torch.randn(16, H, device="cuda").bfloat16(), torch.randn(16, H, device="cuda").bfloat16()
    w, b = torch.randn(H, device="cuda").bfloat16(), torch.randn(H, device="cuda").bfloat16()

    def want():
        st.set_call_id(3)
        return (dropout(x, 0.25).float() + r.float()).bfloat16()

    st.set_call_id(3)
    y, z = fused_norm(x, w, b, r, EPS, False, 0.25)
    assert torch.equal(z, want())
    assert torch.allclose(y.float(), _norm(z.float(), w.float(), b.float(), False), atol=0.05, rtol=2.0 ** -7)
    graph = torch.cuda.CUDAGraph()
    st.set_call_id(3)
    with torch.cuda.graph(graph):
        captured = fused_norm(x, w, b, r, EPS, False, 0.25)[1]
    for _ in range(2):
        graph.replay()
        assert torch.equal(captured, want())
        st.advance_micro()
    graph.replay()
    assert torch.equal(captured, want()) and not torch.equal(captured, z)
