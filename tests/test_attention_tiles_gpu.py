"""Flash attention forward at the edges of its 128 x 128 blocks, and with row maxima that grow from block to block
(the output accumulator is rescaled in place), against fp64 PyTorch; rotary embedding folded into the packed form."""
import math

import pytest
import torch

from merak_b200.ops import _lib
from merak_b200.ops.attention import flash_attention, rope_attention_packed
from merak_b200.ops.elementwise import apply_rope, rope_tables

pytestmark = pytest.mark.gpu


def _ref(q, k, v, bias, causal):
    q, k, v = (t.double().transpose(1, 2) for t in (q, k, v))
    rep = q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1)
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    if bias is not None:
        # a mask of the lowest fp32 value overflows to -inf in the kernels' log2 units: such keys are invisible
        s = s + bias.double().masked_fill(bias < -1e30, float("-inf"))[:, None, None]
    if causal:
        keep = torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).tril(s.shape[-1] - s.shape[-2])
        s = s.masked_fill(~keep, float("-inf"))
    p = torch.nan_to_num(torch.softmax(s, -1), nan=0.0)          # rows without a visible key give zeros
    return (p @ v).transpose(1, 2)


@pytest.mark.parametrize("Lq,Lk", [(1, 1), (1, 129), (127, 128), (128, 127), (129, 257), (300, 100), (257, 640)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("growth", [0.0, 40.0, -40.0])
def test_forward(Lq, Lk, D, causal, growth):
    torch.manual_seed(Lq * 1000 + Lk)
    q = torch.randn(2, Lq, 4, D, device="cuda").bfloat16()
    k = torch.randn(2, Lk, 2, D, device="cuda").bfloat16()
    v = torch.randn(2, Lk, 2, D, device="cuda").bfloat16()
    bias = None
    if growth:      # scores rise (or fall) by `growth` over the keys; the first keys are masked out altogether
        bias = torch.linspace(0, growth, Lk, device="cuda").repeat(2, 1)
        bias[1, :Lk // 2] = torch.finfo(torch.float32).min
    out = flash_attention(q, k, v, key_bias=bias, causal=causal)
    torch.cuda.synchronize()
    _lib.assert_status_ok("attention")
    ref = _ref(q, k, v, bias, causal)
    # probabilities and outputs are rounded to bf16 once each (2^-9), sums are fp32
    assert (out.double() - ref).norm() <= 2.0 ** -7 * ref.norm() + 1e-6


@pytest.mark.parametrize("hq,hkv,D", [(4, 4, 64), (4, 2, 128), (3, 1, 128)])
@pytest.mark.parametrize("L", [1, 77, 129])
@pytest.mark.parametrize("given_positions", [False, True])
def test_rope_attention_packed(hq, hkv, D, L, given_positions):
    torch.manual_seed(L)
    base = torch.randn(2, L, hq + 2 * hkv, D, device="cuda").bfloat16()
    cos, sin = rope_tables(256, D, device="cuda")
    pos = torch.randint(0, 256, (2, L), device="cuda") if given_positions else None
    a, b = base.clone().requires_grad_(True), base.clone().requires_grad_(True)
    out = rope_attention_packed(a, hq, hkv, cos, sin, pos)
    q, k, v = b[:, :, :hq], b[:, :, hq:hq + hkv], b[:, :, hq + hkv:]
    want = flash_attention(apply_rope(q, cos, sin, pos), apply_rope(k, cos, sin, pos), v, causal=True)
    assert torch.equal(out, want)
    g = torch.randn_like(out)
    out.backward(g)
    want.backward(g)
    # dQ is summed with atomics (fp32) in both, everything else is the same arithmetic
    assert (a.grad.float() - b.grad.float()).norm() <= 2.0 ** -8 * b.grad.float().norm()
    assert torch.equal(a.grad[:, :, hq + hkv:], b.grad[:, :, hq + hkv:])


def _blockwise(q, k, v, causal):
    """The kernel's roundings and no others, sums in fp64: P in bf16 relative to the running row maximum over blocks of
    128 keys, the output in bf16."""
    q, k, v = (t.double().transpose(1, 2) for t in (q, k, v))
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    if causal:
        s = s.masked_fill(~torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).tril(), float("-inf"))
    m = torch.full_like(s[..., :1], float("-inf"))
    l, o = torch.zeros_like(m), torch.zeros_like(q)
    for j in range(0, s.shape[-1], 128):
        new = torch.maximum(m, s[..., j:j + 128].amax(-1, keepdim=True))
        p, alpha = torch.exp(s[..., j:j + 128] - new), torch.exp(m - new)
        l, o = l * alpha + p.sum(-1, keepdim=True), o * alpha + p.bfloat16().double() @ v[..., j:j + 128, :]
        m = new
    return (o / l).transpose(1, 2).bfloat16()


@pytest.mark.parametrize("L", [512, 1001])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("spread", [1.0, 3.0])
def test_forward_precision(L, D, causal, spread):
    """No further from fp64 than the roundings of P and of the output account for.  Peaked rows tell a maximum in use
    that is not the row's own: their largest probability is then no longer exact in bf16."""
    torch.manual_seed(L + D)
    q = (torch.randn(2, L, 4, D, device="cuda") * spread).bfloat16()
    k, v = (torch.randn(2, L, 4, D, device="cuda").bfloat16() for _ in range(2))
    out = flash_attention(q, k, v, causal=causal)
    ref = _ref(q, k, v, None, causal)
    err, floor = (out.double() - ref).norm(), (_blockwise(q, k, v, causal).double() - ref).norm()
    # the same roundings of nearly the same numbers; few of the 2^18 or more flip with exp2f's last bit
    assert err <= 1.02 * floor, (err / floor).item()


@pytest.mark.parametrize("L", [128, 300])
@pytest.mark.parametrize("scale", [-2.0, 0.0, 2.0])
@pytest.mark.parametrize("dropout_p", [0.0, 1e-7])
def test_forward_scale_of_any_sign(L, scale, dropout_p):
    """Scores some hundreds wide: probabilities relative to anything but the row's maximum overflow."""
    torch.manual_seed(L)
    q, k, v = (torch.randn(1, L, 2, 64, device="cuda").bfloat16() for _ in range(3))
    out = flash_attention(4 * q, 4 * k, v, scale=scale, dropout_p=dropout_p)     # at 1e-7 no probability is dropped
    ref = _ref(4 * q * (scale * 8.0), 4 * k, v, None, False)                     # (the oracle divides by 8)
    assert (out.double() - ref).norm() <= 2.0 ** -7 * ref.norm()


def test_rope_attention_packed_at_an_odd_address():
    cos, sin = rope_tables(64, 64, device="cuda")
    base = torch.randn(1 + 2 * 37 * 12 * 64, device="cuda").bfloat16()
    odd = base[1:].view(2, 37, 12, 64).requires_grad_(True)
    even = odd.detach().clone().requires_grad_(True)
    g = torch.randn(2, 37, 4, 64, device="cuda").bfloat16()
    outs = [rope_attention_packed(t, 4, 4, cos, sin) for t in (odd, even)]
    for o in outs:
        o.backward(g)
    assert torch.equal(*outs) and (odd.grad.float() - even.grad.float()).norm() <= 2.0 ** -8 * even.grad.float().norm()
