"""Next-token cross entropy on unsliced logits, and rows without a target, against PyTorch in fp32."""
import pytest
import torch
import torch.nn.functional as F

from merak_b200.ops.cross_entropy import next_token_cross_entropy, softmax_cross_entropy

pytestmark = pytest.mark.gpu


def _pitched(x):
    """The same values with rows padded to 16 bytes, as the GEMM writes logits of a ragged vocabulary."""
    pitch = (x.shape[-1] + 7) // 8 * 8
    buf = torch.zeros(*x.shape[:-1], pitch, dtype=x.dtype, device=x.device)
    buf[..., :x.shape[-1]] = x
    return buf[..., :x.shape[-1]]


@pytest.mark.parametrize("B,L,V", [(2, 2, 8), (3, 5, 1001), (1, 129, 2048), (4, 33, 50257)])
@pytest.mark.parametrize("pitched", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_next_token_matches_sliced(B, L, V, pitched, dtype):
    torch.manual_seed(B * L + V)
    base = torch.randn(B, L, V, device="cuda").to(dtype)
    logits = (_pitched(base) if pitched else base).detach().requires_grad_(True)
    labels = torch.randint(0, V, (B, L), device="cuda")
    if L > 2:
        labels[0, 1] = -100
    loss = next_token_cross_entropy(logits, labels)
    loss.backward()
    ref_in = base.float().clone().requires_grad_(True)
    ref = F.cross_entropy(ref_in[:, :-1].reshape(-1, V), labels[:, 1:].reshape(-1))
    ref.backward()
    # fp32 sums over a row; the gradient leaves in the dtype of the logits (bf16: 2^-9 of each value)
    assert abs(loss.item() - ref.item()) < 1e-5 * max(1.0, abs(ref.item()))
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
    assert (logits.grad.float() - ref_in.grad).norm() <= tol * ref_in.grad.norm()
    assert torch.count_nonzero(logits.grad[:, -1]) == 0


def test_short_or_odd_inputs_take_the_sliced_path():
    logits = torch.randn(2, 4, 16, device="cuda", dtype=torch.bfloat16)
    labels = torch.randint(0, 16, (2, 5), device="cuda")[:, :4]
    assert torch.equal(next_token_cross_entropy(logits, labels),
                       softmax_cross_entropy(logits[:, :-1], labels[:, 1:]))


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rows_without_target_are_not_read(bad, dtype):
    logits = torch.randn(6, 43, device="cuda").to(dtype)
    labels = torch.tensor([1, -100, 42, 0, -100, 5], device="cuda")
    clean = _pitched(logits).detach().requires_grad_(True)
    a = softmax_cross_entropy(clean, labels)
    a.backward()
    logits[1], logits[4] = bad, bad
    dirty = _pitched(logits).detach().requires_grad_(True)
    b = softmax_cross_entropy(dirty, labels)
    b.backward()
    assert torch.equal(a, b) and torch.equal(clean.grad, dirty.grad)


def test_no_row_has_a_target():
    logits = torch.randn(3, 16, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    loss = softmax_cross_entropy(logits, torch.full((3,), -100, device="cuda"))
    loss.backward()
    assert loss.item() == 0.0 and torch.count_nonzero(logits.grad) == 0


@pytest.mark.parametrize("offset", [1, 4, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_logits_that_start_inside_a_row(offset, dtype):
    """A slice of the vocabulary: rows 16-byte pitched, the first of them not 16-byte aligned (but at offset 8)."""
    B, L, V = 3, 5, 1001
    torch.manual_seed(offset)
    wide = torch.randn(B, L, 1016, device="cuda").to(dtype).requires_grad_(True)
    labels = torch.randint(0, V, (B, L), device="cuda")
    ref_in = wide.detach().float()[..., offset:offset + V].requires_grad_(True)
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
    for loss_fn, ref in ((next_token_cross_entropy, F.cross_entropy(ref_in[:, :-1].reshape(-1, V), labels[:, 1:].reshape(-1))),
                         (softmax_cross_entropy, F.cross_entropy(ref_in.reshape(-1, V), labels.reshape(-1)))):
        wide.grad = ref_in.grad = None
        loss = loss_fn(wide[..., offset:offset + V], labels)
        loss.backward()
        ref.backward()
        assert abs(loss.item() - ref.item()) < 1e-5 * abs(ref.item())
        assert (wide.grad[..., offset:offset + V].float() - ref_in.grad).norm() <= tol * ref_in.grad.norm()


@pytest.mark.parametrize("dtype", [torch.bool, torch.uint8, torch.int8, torch.int32, torch.float32])
def test_label_types(dtype):
    """Labels of any type that the cross entropy takes, those too that cannot hold the "no target" value."""
    torch.manual_seed(0)
    logits = torch.randn(2, 7, 64, device="cuda", dtype=torch.bfloat16)
    labels = torch.randint(0, 2 if dtype == torch.bool else 64, (2, 7), device="cuda").to(dtype)
    got, want = next_token_cross_entropy(logits, labels), softmax_cross_entropy(logits[:, :-1], labels[:, 1:])
    assert abs(got.item() - want.item()) < 1e-5 * abs(want.item())      # the same rows, summed in another order


def test_labels_of_another_shape_take_the_sliced_path():
    torch.manual_seed(0)
    logits = torch.randn(2, 4, 16, device="cuda").bfloat16().requires_grad_(True)
    labels = torch.randint(0, 16, (2, 4, 1), device="cuda")
    loss = next_token_cross_entropy(logits, labels)
    loss.backward()
    want = F.cross_entropy(logits[:, :-1].float().reshape(-1, 16), labels[:, 1:].reshape(-1))
    assert abs(loss.item() - want.item()) < 1e-5 and torch.count_nonzero(logits.grad[:, -1]) == 0
