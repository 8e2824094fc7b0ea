"""The one-kernel sampler ends a search over a list of at most 2,048 keys: the same tokens, bit for bit, as the form that passes
over the vocabulary for every digit (whole-number sums, so there is nothing to tolerate).  Rows with three or more NaN or +inf are left out: their
weights make the sums wrap around, which the two forms do not do alike."""
import pytest
import torch

from rust_inference_b200 import ops

pytestmark = pytest.mark.gpu

KINDS = ["normal", "flat", "narrow", "wide", "masked", "equal_pairs"]


def _logits(kind, rows, vocab, g):
    x = torch.randn((rows, vocab), generator=g, device="cuda")
    if kind == "flat":
        return torch.full_like(x, 0.75)
    if kind == "narrow":
        return 3.0 + 1e-3 * x
    if kind == "wide":
        return 40.0 * x
    x = 2.5 * x
    if kind == "masked":
        x[:, 37:] = -float("inf")
    if kind == "equal_pairs":
        x = (x * 8).round() / 8
    return x


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rows,vocab", [(1, 32000), (9, 151936), (37, 50257)])
def test_lists_choose_what_the_passes_choose(kind, rows, vocab, monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(rows * 1000 + len(kind))
    logits = _logits(kind, rows, vocab, g)
    temperature = torch.rand(rows, generator=g, device="cuda") * 1.5 + 0.2
    temperature[rows // 2] = 0.0 if rows > 1 else 1.0
    # edges of a list: exactly full, one too many, nothing, all
    ks = torch.tensor([0, 1, 50, 1500, 2047, 2048, 2049, 6000, vocab], dtype=torch.int32, device="cuda")
    ps = torch.tensor([1.0, 0.9, 1e-7, 0.5, 0.9999, 0.0, 0.05], device="cuda")
    for shift in range(3):
        top_k = ks[(torch.arange(rows, device="cuda") + 3 * shift) % len(ks)].contiguous()
        top_p = ps[(torch.arange(rows, device="cuda") + shift) % len(ps)].contiguous()
        u = torch.rand(rows, generator=g, device="cuda")
        for k, p in ((top_k, top_p), (top_k, None), (None, top_p), (None, None)):
            monkeypatch.setattr(ops, "SAMPLE_ONE_KERNEL", True)
            got = ops.sample(logits, temperature, u, top_k=k, top_p=p)
            monkeypatch.setattr(ops, "SAMPLE_ONE_KERNEL", False)
            want = ops.sample(logits, temperature, u, top_k=k, top_p=p)
            assert torch.equal(got, want), (shift, k is not None, p is not None)


@pytest.mark.parametrize("nans, infs", [(1, 0), (2, 0), (0, 1), (0, 2), (2, 1)])
def test_one_or_two_values_that_are_not_finite(nans, infs, monkeypatch):
    """Their weights are 2^63: sums of up to two of them are the same in both forms (from three on they are not)."""
    rows, vocab = 16, 50257
    g = torch.Generator(device="cuda").manual_seed(10 * nans + infs)
    logits = torch.randn((rows, vocab), generator=g, device="cuda") * 2.5
    for row in logits:
        at = torch.randperm(vocab, generator=g, device="cuda")
        row[at[:nans]] = float("nan")
        row[at[nans:nans + infs]] = float("inf")
    temperature, u = torch.full((rows,), 0.7, device="cuda"), torch.rand(rows, generator=g, device="cuda")
    for k, p in ((0, 1.0), (50, 1.0), (0, 0.9), (50, 0.9), (3000, 0.9)):
        top_k, top_p = torch.full((rows,), k, dtype=torch.int32, device="cuda"), torch.full((rows,), p, device="cuda")
        got = []
        for one in (True, False):
            monkeypatch.setattr(ops, "SAMPLE_ONE_KERNEL", one)
            got.append(ops.sample(logits, temperature, u, top_k=top_k, top_p=top_p, uses_top_k=k > 0, uses_top_p=p < 1.0))
        assert torch.equal(*got), (k, p)
