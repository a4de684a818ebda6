"""Tile widths of the CTA-pair GEMM: whole, halved and strip units, each epilogue through the per-warp boxes, against
fp32 PyTorch.  The sizes give tile counts just above a multiple of the clusters and right edges in every part of a
tile."""
import pytest
import torch

from merak_b200.ops import _lib, gemm as G
from merak_b200.ops.linear import linear, linear_fork

pytestmark = pytest.mark.gpu

SIZES = [(129, 136, 72), (257, 320, 64), (462, 768, 200), (2560, 2304, 64), (2433, 2376, 136), (5000, 1160, 64),
         (3003, 2048, 328), (300, 50257, 64), (1600, 1600, 512)]


def _inputs(M, N, K, a_mn, b_mn):
    torch.manual_seed(M + N + K)
    a = torch.randn((K, M) if a_mn else (M, K), device="cuda").bfloat16()
    b = (torch.randn((K, N) if b_mn else (N, K), device="cuda") * 0.1).bfloat16()
    A, B = (a.float().t() if a_mn else a.float()), (b.float() if b_mn else b.float().t())
    return a, b, A.double() @ B.double()


def _check(out, ref, tol):
    torch.cuda.synchronize()
    _lib.assert_status_ok("gemm")
    err = (out.double() - ref).norm() / ref.norm()
    assert err < tol, err.item()


# bf16 outputs carry 2^-9 of rounding each (2-norm: below 2^-9); fp32 sums of K products below 1e-5
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("layout", [(False, False), (False, True), (True, True)])
def test_bf16_output(size, layout):
    M, N, K = size
    a, b, ref = _inputs(M, N, K, *layout)
    out, _ = G.gemm(a, b, a_mn=layout[0], b_mn=layout[1], block_n=512)
    _check(out, ref, 2.0 ** -8)


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("bias_dtype", [torch.bfloat16, torch.float32])
def test_bias_activation_residual(size, bias_dtype):
    M, N, K = size
    a, b, ref = _inputs(M, N, K, False, False)
    bias = torch.randn(N, device="cuda").to(bias_dtype)
    aux = torch.randn(M, (N + 7) // 8 * 8, device="cuda").bfloat16()[:, :N]
    out, _ = G.gemm(a, b, bias=bias, aux_in=aux, aux_mode=G.AUX_ADD, block_n=512)
    _check(out, ref + bias.double() + aux.double(), 2.0 ** -8)
    out, pre = G.gemm(a, b, bias=bias, act=G.ACT_RELU, want_preact=True, block_n=512)
    _check(pre, ref + bias.double(), 2.0 ** -8)
    _check(out, (ref + bias.double()).clamp(min=0), 2.0 ** -8)


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("accumulate", [False, True])
def test_fp32_output(size, accumulate):
    M, N, K = size
    a, b, ref = _inputs(M, N, K, True, True)
    out = torch.randn(M, (N + 7) // 8 * 8, device="cuda")[:, :N]
    want = ref + out.double() if accumulate else ref
    G.gemm(a, b, a_mn=True, b_mn=True, out=out, accumulate=accumulate, block_n=512)
    _check(out, want, 1e-5)


def _side(M, N, kind):
    """A side tensor in each form that 16-byte accesses do not fit, and in the one that they do."""
    if kind == "aligned":
        return torch.randn(M, (N + 7) // 8 * 8, device="cuda").bfloat16()[:, :N]
    if kind == "pitch":
        pitch = (N + 3) // 4 * 4 + (4 if (N + 3) // 4 % 2 == 0 else 0)             # a multiple of 4, not of 8
        return torch.randn(M, pitch, device="cuda").bfloat16()[:, :N]
    return torch.randn(M, (N + 16) // 8 * 8, device="cuda").bfloat16()[:, 1:N + 1]


SIDE_SIZES = [(129, 136, 72), (257, 300, 64), (462, 772, 200), (2433, 2372, 72), (300, 161, 64)]


@pytest.mark.parametrize("size", SIDE_SIZES)
@pytest.mark.parametrize("kind", ["aligned", "pitch", "pointer"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_side_input(size, kind, dtype):
    M, N, K = size
    a, b, ref = _inputs(M, N, (K + 7) // 8 * 8, False, False)
    aux = _side(M, N, kind)
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
    out, _ = G.gemm(a, b, aux_in=aux, aux_mode=G.AUX_ADD, out_dtype=dtype, block_n=512)
    _check(out, ref + aux.double(), tol)
    out, _ = G.gemm(a, b, act=G.ACT_RELU, aux_in=aux, aux_mode=G.AUX_DACT, out_dtype=dtype, block_n=512)
    _check(out, ref * (aux > 0), tol)


@pytest.mark.parametrize("size", SIDE_SIZES)
@pytest.mark.parametrize("pitch,shift", [(8, 0), (4, 0), (8, 1)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_side_output_stays_in_its_rows(size, pitch, shift, dtype):
    """The pre-activation goes into rows of N values; what lies between and behind them keeps its value."""
    M, N, K = size
    a, b, ref = _inputs(M, N, K, False, False)
    ld = (N + shift + pitch - 1) // pitch * pitch
    ld += 4 if pitch == 4 and ld % 8 == 0 else 0
    buf = torch.full((M * ld + 64,), -7.0, device="cuda", dtype=torch.bfloat16)
    pre = buf[shift:shift + M * ld].view(M, ld)
    out = torch.empty(M, (N + 7) // 8 * 8, device="cuda", dtype=dtype)
    flags = G._F_OUT_F32 if dtype == torch.float32 else 0
    rc = _lib.kernels().mrk_gemm_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0),
                                      out.stride(0), 0, 0, 0, pre.data_ptr(), ld, G.ACT_RELU, G.AUX_NONE, flags, 1.0,
                                      512, _lib.stream_ptr())
    _lib.check(rc, "mrk_gemm_bf16")
    _check(pre[:, :N], ref, 2.0 ** -8)
    _check(out[:, :N], ref.clamp(min=0), 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5)
    assert bool((pre[:, N:] == -7.0).all()) and bool((buf[shift + M * ld:] == -7.0).all()) and bool((buf[:shift] == -7.0).all())


def test_linear_with_unpadded_residual():
    """A residual, and the gradient a fork hands back, whose rows are not multiples of 16 bytes."""
    torch.manual_seed(0)
    x = torch.randn(257, 300, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn(300, 300, device="cuda") * 0.1).bfloat16().requires_grad_(True)
    r = torch.randn(257, 300, device="cuda").bfloat16()
    _check(linear(x, w, None, r).detach(), x.double() @ w.double().t() + r.double(), 2.0 ** -8)
    y, x2 = linear_fork(x, w)
    (y.float().sum() + (x2.float() * r.float()).sum()).backward()
    _check(x.grad, torch.ones(257, 300, device="cuda").double() @ w.detach().double() + r.double(), 2.0 ** -8)
