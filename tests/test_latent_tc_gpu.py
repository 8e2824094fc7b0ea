"""Prefill attention over latent rows of 256 elements whose first elements are the values, on the tcgen05 kernel: against plain
softmax attention in float64, at the edges of query tiles, key blocks, pages and windows."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


# (tokens before, new tokens) of each sequence
@pytest.mark.parametrize("lens", [[(0, 1), (0, 2)], [(0, 127)], [(0, 128), (5, 129)], [(0, 257), (31, 64), (0, 33)], [(700, 300)], [(0, 1100)], [(1000, 3), (0, 500)]])
@pytest.mark.parametrize("H, KV, v_dims, window, sink", [(3, 1, 192, 0, False), (4, 2, 128, 70, True), (2, 1, 40, 1, False), (5, 1, 190, 256, True)])
def test_latent_rows_against_plain_attention(lens, H, KV, v_dims, window, sink):
    from rust_inference_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(sum(a + b for a, b in lens) + H)
    D, page = 256, 32
    pages_of = [-(-(a + b) // page) for a, b in lens]
    total = sum(pages_of) + 3
    order = torch.randperm(total, generator=g, device=DEV).tolist()
    pool = torch.full((total, KV, page, D), float("nan"), dtype=torch.bfloat16, device=DEV)      # what no key lies in is not read as one
    table = torch.full((len(lens), max(pages_of) + 1), -1, dtype=torch.int32, device=DEV)
    start, rows = [0], []
    for b, (past, new) in enumerate(lens):
        n = past + new
        row = (torch.randn((n, KV, D), generator=g, device=DEV) * 0.7).to(torch.bfloat16)
        for p in range(pages_of[b]):
            page_id = order.pop()
            table[b, p] = page_id
            part = row[p * page:(p + 1) * page]
            pool[page_id, :, :len(part)] = part.transpose(0, 1)
        rows.append(row.double())
        start.append(start[-1] + new)
    q = torch.randn((start[-1], H, D), generator=g, device=DEV).to(torch.bfloat16)
    s = torch.randn((H,), generator=g, device=DEV) if sink else None
    scale = 0.08
    got = ops.attention_prefill(q, pool, pool, table, _i32(list(range(len(lens)))), _i32(start), _i32([a + b for a, b in lens]),
                                max(b for _, b in lens), scale, window, sink=s, v_dims=v_dims)
    assert int(ops.error_flag(DEV).item()) == 0
    for b, (past, new) in enumerate(lens):
        i = torch.arange(past, past + new, device=DEV)[:, None]
        j = torch.arange(past + new, device=DEV)[None, :]
        hidden = (j > i) | ((i - j >= window) if window else (j > i))
        for h in range(H):
            k = rows[b][:, h * KV // H]
            score = (q[start[b]:start[b + 1], h].double() @ k.t() * scale).masked_fill(hidden, -math.inf)
            if sink:
                p = torch.softmax(torch.cat([score, s[h].double().expand(new, 1)], dim=1), dim=1)[:, :-1]
            else:
                p = torch.softmax(score, dim=1)
            want = p @ k[:, :v_dims]
            diff = (got[start[b]:start[b + 1], h, :v_dims].double() - want).abs()
            # weights rounded to 8 bits (their sum is not), the result once more: 2^-8 of the weighted magnitudes, twice
            assert (diff <= 2.0 ** -7 * (p @ k[:, :v_dims].abs()) + 1e-5).all(), (b, h)
    assert torch.isfinite(got[..., :v_dims].float()).all()


# forms that the kernel above does not take; kept keys, which count beside a window only; more tokens announced than there are
@pytest.mark.parametrize("form", [dict(window=33, keep=40), dict(chunk=50, keep=3), dict(scale=0.0), dict(scale=-0.05), dict(max_new=500)])
def test_other_forms_against_plain_attention(form):
    from rust_inference_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(7)
    n, H, v_dims = 170, 3, 192
    row = (torch.randn((n, 256), generator=g, device=DEV) * 0.7).to(torch.bfloat16)
    pool = torch.zeros((6, 1, 32, 256), dtype=torch.bfloat16, device=DEV)
    pool.view(192, 256)[:n] = row
    q = torch.randn((n, H, 256), generator=g, device=DEV).to(torch.bfloat16)
    args = {**dict(max_new=n, scale=0.08, window=0, v_dims=v_dims), **form}
    got = ops.attention_prefill(q, pool, pool, _i32([list(range(6))]), _i32([0]), _i32([0, n]), _i32([n]), **args)
    assert int(ops.error_flag(DEV).item()) == 0
    i, j = torch.arange(n, device=DEV)[:, None], torch.arange(n, device=DEV)[None, :]
    inside = i - j < form["window"] if "window" in form else i // form["chunk"] == j // form["chunk"] if "chunk" in form else j >= 0
    seen = (j <= i) & (inside | (j < form.get("keep", 0) if "window" in form else inside))
    k = row.double()
    for h in range(H):
        p = torch.softmax((q[:, h].double() @ k.t() * args["scale"]).masked_fill(~seen, -math.inf), dim=1)
        diff = (got[:, h, :v_dims].double() - p @ k[:, :v_dims]).abs()
        assert (diff <= 2.0 ** -7 * (p @ k[:, :v_dims].abs()) + 1e-5).all(), h      # the bound of the test above
