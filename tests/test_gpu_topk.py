"""The exact top-k against a full sort: value descending, then lower id."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 16, 64])
@pytest.mark.parametrize("kind", ["random", "ties", "one level", "a low group", "runs", "infinities"])
@pytest.mark.parametrize("vocab", [64, 300, 4096, 4106, 151936])
def test_topk_is_the_head_of_a_full_sort(vocab, kind, count):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(vocab + count)
    x = torch.randn(5, vocab, device="cuda", generator=g)
    ids = torch.arange(vocab, device="cuda")
    if kind == "ties":
        x = (x * 2).round() + 0.0             # (no -0)
    elif kind == "one level":
        x = torch.ones_like(x)
    elif kind == "a low group":                # more keys pass than the list of candidates holds
        x[:, ids % 256 < 4] = -1e30
    elif kind == "runs":
        x = x.sort(-1).values
    elif kind == "infinities":
        x[:, ::3] = float("-inf")
        x[:, 5] = float("inf")
    got_i, got_v = torch.zeros(5, count, dtype=torch.int32, device="cuda"), torch.zeros(5, count, device="cuda")
    K.topk(x, count, K.topk_scratch(5, vocab, count), got_i, got_v)
    v, i = x.sort(dim=-1, descending=True, stable=True)
    assert torch.equal(got_i.long(), i[:, :count]) and torch.equal(got_v, v[:, :count])


@pytest.mark.parametrize("count", [2, 3])                   # the last count that is found by rounds, the first by the threshold
@pytest.mark.parametrize("vocab", [3, 300, 151936])
def test_topk_on_both_sides_of_the_forms(vocab, count):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    x = (torch.randn(7, vocab, device="cuda", generator=torch.Generator(device="cuda").manual_seed(vocab)) * 3).round() + 0.0
    got_i, got_v = torch.zeros(7, count, dtype=torch.int32, device="cuda"), torch.zeros(7, count, device="cuda")
    K.topk(x, count, K.topk_scratch(7, vocab, count), got_i, got_v)
    v, i = x.sort(dim=-1, descending=True, stable=True)
    assert torch.equal(got_i.long(), i[:, :count]) and torch.equal(got_v, v[:, :count])
