"""The forms of the kernels between the products that take whole pieces of rows, at the edges of their pieces and tokens, against
float64 and against the forms that take an element at a time (rows that do not start on whole pieces)."""
import numpy as np
import pytest
import torch

from rust_inference_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
TOL = {"float32": 2e-6, "bfloat16": 5e-3}      # float32 functions; one rounding to 8 bits


def _i32(v):
    return torch.tensor(np.asarray(v, dtype=np.int32), device=DEV)


def _rand(seed, *shape):
    return torch.randn(shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


def _close(got, want, tol):
    assert ((got.double() - want.double()).norm() / want.double().norm()).item() <= tol


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tokens, heads, vdim", [(1, 1, 4), (3, 5, 96), (700, 16, 128), (7, 3, 132), (2, 2, 256), (5, 2, 260), (9, 4, 66)])
@pytest.mark.parametrize("fn", ["silu", "sigmoid"])
def test_head_norm_gate(tokens, heads, vdim, fn, dtype):
    o, gain = _rand(1, tokens, heads, vdim), 1 + 0.1 * _rand(2, vdim)
    wide = _rand(3, tokens, heads * vdim + 8).to(DT[dtype])
    for g in (wide[:, 8:], wide[:, 4:4 + heads * vdim], wide[:, 1:1 + heads * vdim]):       # the last: element by element
        z = g.double().view(tokens, heads, vdim)
        want = o.double() / torch.sqrt((o.double() ** 2).mean(-1, keepdim=True) + 1e-6) * gain.double() * torch.sigmoid(z) * (z if fn == "silu" else 1)
        _close(ops.head_norm_gate(o, gain, 1e-6, g, DT[dtype], fn).view(tokens, heads, vdim), want, TOL[dtype])


def _at_odd_place(t):
    """The same values as a block of columns that starts one element behind a whole piece."""
    wide = torch.empty((t.shape[0], t.shape[1] + 5), dtype=t.dtype, device=DEV)
    wide[:, 1:1 + t.shape[1]] = t
    return wide[:, 1:1 + t.shape[1]]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tokens, heads, vdim", [(1, 1, 4), (3, 5, 96), (700, 16, 128), (70, 3, 132), (40, 2, 256)])
def test_head_norm_gate_gives_the_bits_of_a_column_at_a_time(tokens, heads, vdim, dtype):
    o, gain, g = _rand(15, tokens, heads, vdim), 1 + 0.1 * _rand(16, vdim), _rand(17, tokens, heads * vdim).to(DT[dtype])
    for fn in ("silu", "sigmoid"):
        assert torch.equal(ops.head_norm_gate(o, gain, 1e-6, g, DT[dtype], fn), ops.head_norm_gate(o, gain, 1e-6, _at_odd_place(g), DT[dtype], fn))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tokens, H, G, dim", [(1, 2, 1, 4), (3, 4, 2, 36), (300, 4, 4, 128), (65, 2, 1, 132), (257, 2, 2, 260), (7, 2, 1, 512)])
def test_unit_vectors_and_decays_give_the_bits_of_a_channel_at_a_time(tokens, H, G, dim, dtype):
    vdim = 8
    qkv = _rand(18, tokens, 2 * G * dim + H * vdim)
    proj, z = _rand(19, tokens, H).to(DT[dtype]), _rand(20, tokens, H * dim).to(DT[dtype])
    dt_bias, a_log = _rand(21, H * dim), 0.3 * _rand(22, H)
    results = []
    for decays in (z, _at_odd_place(z)):                      # the second: a channel at a time
        q, state = qkv.clone(), _rand(23, 1, H, dim, vdim)
        o = ops.delta_rule_recurrent(q, 0, G * dim, 2 * G * dim, proj, 0, decays, dt_bias, a_log, dim ** -0.5, state, _i32([0]), _i32([0, tokens]),
                                     H, G, dim, vdim)
        results.append((q, o, state))
    for a, b in zip(*results):
        assert torch.equal(a, b)


# steps of many elements take four tokens a thread; sequences that begin and end anywhere in a thread's four, of one and two tokens too
@pytest.mark.parametrize("C", [72, 12296])
@pytest.mark.parametrize("lens", [[256], [259], [1, 2, 3, 250, 1, 1, 4], [64] * 5, [255, 2]])
def test_short_conv_over_many_tokens(lens, C):
    T, slots = sum(lens), len(lens) + 2
    x = _rand(4, T, C + 8).bfloat16()[:, :]
    w = 0.5 * _rand(5, C, 4)
    wt = w.t().contiguous()
    state = _rand(6, slots, 3, C)
    order = list(range(len(lens)))[::-1]
    args = (_i32(np.repeat(np.arange(len(lens)), lens)), _i32(order), _i32(np.concatenate([[0], np.cumsum(lens)])))
    a, b = state.clone(), state.clone()
    got = ops.short_conv(x, 8, w, a, *args, weight_t=wt)
    assert torch.equal(got, ops.short_conv(x, 8, w, b, *args)) and torch.equal(a, b)             # an element at a time
    start = np.concatenate([[0], np.cumsum(lens)])
    for i, n in enumerate(lens):
        seq = torch.cat([state[order[i]].double(), x[start[i]:start[i + 1], 8:].double()])
        z = sum(w[:, j].double() * seq[j:j + n] for j in range(4))
        _close(got[start[i]:start[i + 1]], z * torch.sigmoid(z), 1e-6)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tokens, H, dim, rot, rank, row", [(1, 1, 8, 8, 8, 16), (3, 5, 16, 24, 40, 64), (300, 7, 128, 64, 192, 256), (260, 32, 8, 8, 248, 272),
                                                            (5, 3, 12, 4, 20, 32)])
def test_latent_rows(tokens, H, dim, rot, rank, row, dtype):
    dt, page = DT[dtype], 32
    pages = -(-tokens // page)
    cols = H * (dim + rot) + rank + rot
    table = _rand(7, tokens, rot // 2, 2)
    gain = 1 + 0.1 * _rand(8, rank)
    base = _rand(9, tokens, cols + 9).to(dt)
    qa = _rand(10, tokens, H, rank).to(dt)
    meta = (_i32([range(pages)]), _i32([0] * tokens), _i32(range(tokens)), _i32([0]))
    results = []
    for first in (8, 1):                                      # the second: element by element
        proj = torch.zeros((tokens, cols + 16), dtype=dt, device=DEV)
        proj[:, first:first + cols] = base[:, :cols]
        pool = torch.zeros((pages, 1, page, row), dtype=dt, device=DEV)
        qf = ops.latent_prep(proj, first, first + H * (dim + rot), qa, H, dim, rot, rank, gain, 1e-6, table, pool, *meta, row=row)
        results.append((qf, pool))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    q = base[:, :H * (dim + rot)].double().view(tokens, H, dim + rot)[:, :, dim:]
    c, s = table[..., 0].double()[:, None], table[..., 1].double()[:, None]
    u, v = q[..., 0::2], q[..., 1::2]
    want = torch.cat([qa.double(), torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), torch.zeros((tokens, H, row - rank - rot), device=DEV)], -1)
    _close(results[0][0], want, TOL[dtype])


@pytest.mark.parametrize("tokens", [1, 16, 17, 64, 65, 300])
@pytest.mark.parametrize("sets", [[(8, 64, 64)], [(0, 64, 2048), (64, 64, 2048)], [(16, 8, 72), (24, 128, 8)], [(8, 16, 136), (32, 24, 1000)]])
def test_low_rank_products(tokens, sets):
    x = _rand(11, tokens, 160).bfloat16()
    given = [(col, _rand(12 + i, N, K).bfloat16()) for i, (col, K, N) in enumerate(sets)]
    for (col, w), y in zip(given, ops.low_rank(x, *given)):
        want = x[:, col:col + w.shape[1]].double() @ w.double().T
        _close(y, want, 3e-3)                                # one rounding to 8 bits: 2^-9 at most, uniform 2^-9 / sqrt(3)
        assert torch.equal(y, ops.low_rank(x.clone(), (col, w))[0])


# the product's order of sums changes with its kernel: the weight-streaming one up to 12 tokens and for few outputs up to 16, then the
# tcgen05 one, then the library's
@pytest.mark.parametrize("tokens", [1, 8, 12, 13, 16, 17, 32, 33, 65, 1000])
@pytest.mark.parametrize("K, N", [(8, 1024), (24, 2048), (64, 2048), (72, 5000), (128, 1024), (128, 5632)])
def test_low_rank_products_give_the_bits_of_the_product_of_a_copy(tokens, K, N, monkeypatch):
    monkeypatch.setattr(ops, "LOW_RANK_MOST_WORK", (0, 1 << 60, 1 << 60))
    x, w = _rand(24, tokens, 256).bfloat16(), _rand(25, N, K).bfloat16()
    assert torch.equal(ops.low_rank(x, (16, w))[0], ops.linear(x[:, 16:16 + K].contiguous(), w))


def test_low_rank_columns_that_are_not_whole_pieces():
    x, w = _rand(13, 9, 83).bfloat16(), _rand(14, 50, 20).bfloat16()
    _close(ops.low_rank(x, (3, w))[0], x[:, 3:23].double() @ w.double().T, 3e-3)
