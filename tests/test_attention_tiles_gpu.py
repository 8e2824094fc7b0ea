"""The float32 attention over many rows (tiles of 32 rows and strips of 32 keys in registers): bit for bit what the form with a row per
warp gives, which rows of queries that do not start on 16 bytes take, over all kinds of masks, and against float64."""
import numpy as np
import pytest
import torch

from rust_inference_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(v):
    return torch.tensor(np.asarray(v, dtype=np.int32), device=DEV)


def _make(lens, past, H, KV, Dh, page, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    total = [a + b for a, b in zip(lens, past)]
    per = max(-(-t // page) for t in total)
    pages = per * len(lens) + 1
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(seed)).numpy()
    table = order[:per * len(lens)].reshape(len(lens), per)
    k, v = (torch.randn((pages, KV, page, Dh), generator=g, device=DEV) for _ in range(2))
    for b, t in enumerate(total):                              # what nobody wrote must not matter
        for p in range(per):
            n = min(max(t - p * page, 0), page)
            k[table[b, p], :, n:] = float("nan")
            v[table[b, p], :, n:] = float("nan")
    q = torch.randn((sum(lens), H, Dh), generator=g, device=DEV)
    start = np.concatenate([[0], np.cumsum(lens)])
    return q, k, v, (_i32(table), _i32(range(len(lens))), _i32(start), _i32(total)), table, total


def _elsewhere(q):
    """The same queries, not on 16 bytes."""
    other = torch.empty(q.numel() + 1, device=DEV)[1:].view(q.shape)
    other.copy_(q)
    return other


@pytest.mark.parametrize("Dh", [64, 128, 256])
@pytest.mark.parametrize("lens, past, H, KV, page", [
    ([64], [0], 4, 4, 32), ([33, 1, 70], [0, 40, 95], 8, 2, 32), ([200], [0], 16, 2, 64), ([17], [301], 32, 1, 32), ([130, 65], [31, 0], 6, 2, 96),
    ([9], [64], 64, 1, 32)])
@pytest.mark.parametrize("kind", ["plain", "window", "keep", "chunks", "cap and sink", "bias"])
def test_tiles_give_the_bits_of_single_rows(lens, past, H, KV, page, kind, Dh):
    q, k, v, args, table, total = _make(lens, past, H, KV, Dh, page)
    more = {"plain": {}, "window": dict(window=37), "keep": dict(window=37, keep=5), "chunks": dict(chunk=48),
            "cap and sink": dict(softcap=5.0, sink=torch.randn(H, device=DEV)),
            "bias": dict(dist_bias=ops.pad_distance_bias(torch.randn((H, 60), device=DEV)))}[kind]
    got = ops.attention(q, k, v, *args, max(lens), Dh ** -0.5, **more)
    want = ops.attention(_elsewhere(q), k, v, *args, max(lens), Dh ** -0.5, **more)
    assert torch.isfinite(got).all() and torch.equal(got, want)


@pytest.mark.parametrize("Dh", [64, 128, 256])
def test_against_float64(Dh):
    lens, past, H, KV, page = [90, 40], [0, 77], 8, 2, 32
    q, k, v, args, table, total = _make(lens, past, H, KV, Dh, page, seed=3)
    got = ops.attention(q, k, v, *args, max(lens), Dh ** -0.5)
    at = 0
    for b, (n, t) in enumerate(zip(lens, total)):
        kk = k[table[b]].permute(1, 0, 2, 3).reshape(KV, -1, Dh)[:, :t].double().repeat_interleave(H // KV, 0)
        vv = v[table[b]].permute(1, 0, 2, 3).reshape(KV, -1, Dh)[:, :t].double().repeat_interleave(H // KV, 0)
        s = torch.einsum("nhd,hkd->hnk", q[at:at + n].double(), kk) * Dh ** -0.5
        s = s.masked_fill(torch.arange(t, device=DEV) > torch.arange(t - n, t, device=DEV)[:, None], float("-inf"))
        want = torch.einsum("hnk,hkd->nhd", s.softmax(-1), vv)
        assert ((got[at:at + n].double() - want).norm() / want.norm()).item() <= 1e-6
        at += n


def test_values_that_some_rows_do_not_see_may_be_anything():
    q, k, v, args, table, total = _make([60], [0], 4, 1, 64, 32, seed=5)
    v[table[0][1], 0, 8] = float("inf")                       # position 40
    k[table[0][1], 0, 12] = float("nan")                      # position 44
    got = ops.attention(q, k, v, *args, 60, 0.125)
    assert torch.isfinite(got[:40]).all() and not torch.isfinite(got[40:]).all(-1).any()
    again = ops.attention(_elsewhere(q), k, v, *args, 60, 0.125)
    assert torch.equal(torch.nan_to_num(got), torch.nan_to_num(again))
