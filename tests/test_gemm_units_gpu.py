"""Tile widths of the CTA-pair GEMM: whole, halved and strip units, each epilogue through the per-warp boxes, against
fp32 PyTorch.  The sizes give tile counts just above a multiple of the clusters and right edges in every part of a
tile."""
import pytest
import torch

from merak_b200.ops import _lib, gemm as G

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
