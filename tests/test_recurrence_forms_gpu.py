"""The recurrent mixers' kernels in the forms that steps of real sizes take (16-byte copies, rings that wrap, one and two columns a
lane): the same bits for prompts, pieces of prompts and single tokens, and values that are not finite."""
import numpy as np
import pytest
import torch

from rust_inference_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(v):
    return torch.tensor(np.asarray(v, dtype=np.int32), device=DEV)


def _same(a, b):
    """The same numbers, NaN in the same places."""
    return torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))


class Gla:
    """Gated linear attention over the tokens of several sequences, cut into steps; ``ones``: one decay per head and a column of ones."""

    def __init__(self, lens, H, dim, vdim, dtype, ones=False, pad=0, seed=0):
        g = torch.Generator(device=DEV).manual_seed(seed + 31 * sum(lens) + dim)
        self.lens, self.H, self.dim, self.vdim, self.ones, self.pad = lens, H, dim, vdim, ones, pad
        self.width = 2 * H * dim + H * vdim + pad
        self.proj = [torch.randn((n, self.width), generator=g, device=DEV).to(dtype) for n in lens]
        self.z = [(torch.randn((n, H * dim), generator=g, device=DEV) * 2).to(dtype) for n in lens]
        self.gates = [torch.rand((n, H, 3), generator=g, device=DEV) for n in lens]
        self.bias = torch.rand(H * dim, generator=g, device=DEV) * 3
        self.slots = _i32([len(lens) - b for b in range(len(lens))])

    def columns(self):
        return self.pad, self.pad + self.H * self.dim, self.pad + 2 * self.H * self.dim

    def state(self):
        return torch.zeros((len(self.lens) + 2, self.H, self.dim, self.vdim + self.ones), device=DEV)

    def step(self, state, pieces):
        """pieces: (sequence, from, to) of each sequence of the step; its outputs, one tensor per piece."""
        proj = torch.cat([self.proj[b][i:j] for b, i, j in pieces])
        start = np.concatenate([[0], np.cumsum([j - i for _, i, j in pieces])])
        slots, single = self.slots[[b for b, _, _ in pieces]].contiguous(), all(j - i == 1 for _, i, j in pieces)
        if self.ones:
            gates = torch.cat([self.gates[b][i:j] for b, i, j in pieces])
            o = ops.scalar_decay_recurrent(proj, *self.columns(), gates, self.dim ** -0.5, state, slots, _i32(start), self.H, self.dim,
                                           self.vdim, ones=True, single=single)
        else:
            z = torch.cat([self.z[b][i:j] for b, i, j in pieces])
            o = ops.gla_recurrent(proj, *self.columns(), z, self.bias, 16.0, self.dim ** -0.5, state, slots, _i32(start), self.H,
                                  self.dim, self.vdim, single=single)
        return [o[start[k]:start[k + 1]] for k in range(len(pieces))]

    def walk(self, cuts):
        """Every sequence cut where ``cuts`` says, the steps one after the other: outputs per sequence, and the states."""
        state, outs, at = self.state(), [[] for _ in self.lens], 0
        for to in cuts + [max(self.lens)]:
            pieces = [(b, min(at, n), min(to, n)) for b, n in enumerate(self.lens) if min(at, n) < min(to, n)]
            for (b, _, _), o in zip(pieces, self.step(state, pieces) if pieces else []):
                outs[b].append(o)
            at = to
        return [torch.cat(o) for o in outs], state

    def exact(self):
        """Outputs and states in float64 (slots as above)."""
        outs, state = [], self.state().double()
        q_col, k_col, v_col = self.columns()
        for b, n in enumerate(self.lens):
            p = self.proj[b].double()
            q, k = (p[:, c:c + self.H * self.dim].view(n, self.H, self.dim) for c in (q_col, k_col))
            v = p[:, v_col:v_col + self.H * self.vdim].view(n, self.H, self.vdim)
            if self.ones:
                v = torch.cat([v, torch.ones_like(v[..., :1])], dim=-1)
                a, k = self.gates[b][:, :, :1].double().expand_as(k), k * self.gates[b][:, :, 1:2].double()
            else:
                a = torch.sigmoid(self.z[b].double() + self.bias.double()).pow(1 / 16.0).view(n, self.H, self.dim)
            S, o = torch.zeros_like(state[0]), []
            for t in range(n):
                S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
                o.append((S * (q[t] * self.dim ** -0.5)[:, :, None]).sum(1))
            outs.append(torch.stack(o))
            state[int(self.slots[b])] = S
        return outs, state


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("ones", [False, True])
@pytest.mark.parametrize("dim, vdim", [(64, 32), (128, 24)])
def test_an_infinite_last_value_is_infinite_in_every_cutting(dim, vdim, ones, dtype):
    gla = Gla([19, 16, 1], 2, dim, vdim, dtype, ones)
    for p in gla.proj:
        p[-1, -3] = float("inf")                             # the last token's value of one column
    outs, state = gla.walk([])
    singly, state1 = gla.walk(list(range(1, 19)))
    assert all(_same(a, b) for a, b in zip(outs, singly)) and _same(state, state1)
    assert torch.isinf(state).any() and not torch.isnan(state).any()


# 16-byte copies (everything a multiple of eight) and element by element; 3, 4, 13 groups of 16 tokens; a last column on its own
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("ones", [False, True])
@pytest.mark.parametrize("dim, vdim, pad", [(64, 128, 0), (128, 64, 8), (48, 32, 0), (128, 128, 0), (96, 33, 0), (64, 64, 3), (20, 8, 0)])
def test_gla_prompts_pieces_and_single_tokens(dim, vdim, pad, ones, dtype, monkeypatch):
    gla = Gla([47, 200, 1, 48, 65], 2, dim, vdim, dtype, ones, pad)
    outs, state = gla.walk([])
    want, want_state = gla.exact()
    for got, exact in zip(outs + [state], want + [want_state]):
        # float32 sums of up to 200 tokens and 128 channels, decays from float32 exponentials: some 1e-6 of the largest
        assert (got.double() - exact).abs().max() <= 2e-5 * exact.abs().max()
    for cuts in ([], [3, 19, 20, 51, 52, 130], list(range(1, 66)) + [80]):
        if not cuts:                                        # the decays by a kernel of their own
            monkeypatch.setattr(ops, "GLA_OWN_DECAYS", 0)
        pieces, state1 = gla.walk(cuts)
        monkeypatch.undo()
        assert all(torch.equal(a, b) for a, b in zip(pieces, outs)) and torch.equal(state, state1)


class Delta(Gla):
    """The gated delta rule, likewise; ``per_head``: one decay per head."""

    def __init__(self, lens, H, Gq, dim, vdim, dtype, per_head=False, pad=0, seed=0):
        g = torch.Generator(device=DEV).manual_seed(seed + 17 * sum(lens) + dim)
        self.lens, self.H, self.Gq, self.dim, self.vdim, self.ones, self.per_head, self.pad = lens, H, Gq, dim, vdim, False, per_head, pad
        wide = H if per_head else H * dim
        self.qkv = [torch.randn((n, pad + 2 * Gq * dim + H * vdim), generator=g, device=DEV) for n in lens]
        self.proj = [torch.randn((n, H + 3), generator=g, device=DEV).to(dtype) for n in lens]
        self.z = [torch.randn((n, wide), generator=g, device=DEV).to(dtype) for n in lens]
        self.dt_bias = torch.randn(wide, generator=g, device=DEV) - 3
        self.a_log = torch.rand(H, generator=g, device=DEV)
        self.slots = _i32([len(lens) - b for b in range(len(lens))])

    def columns(self):
        return self.pad, self.pad + self.Gq * self.dim, self.pad + 2 * self.Gq * self.dim

    def step(self, state, pieces):
        qkv, proj, z = (torch.cat([x[b][i:j] for b, i, j in pieces]) for x in (self.qkv, self.proj, self.z))
        start = np.concatenate([[0], np.cumsum([j - i for _, i, j in pieces])])
        slots, single = self.slots[[b for b, _, _ in pieces]].contiguous(), all(j - i == 1 for _, i, j in pieces)
        o = ops.delta_rule_recurrent(qkv, *self.columns(), proj, 2, z, self.dt_bias, self.a_log, self.dim ** -0.5, state, slots,
                                     _i32(start), self.H, self.Gq, self.dim, self.vdim, single=single)
        return [o[start[k]:start[k + 1]] for k in range(len(pieces))]

    def exact(self):
        outs, state, H, per = [], self.state().double(), self.H, self.H // self.Gq
        q_col, k_col, v_col = self.columns()
        for b, n in enumerate(self.lens):
            x = self.qkv[b].double()
            q, k = (x[:, c:c + self.Gq * self.dim].view(n, self.Gq, self.dim) for c in (q_col, k_col))
            q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
            q, k = (q * self.dim ** -0.5).repeat_interleave(per, 1), k.repeat_interleave(per, 1)
            v = x[:, v_col:v_col + H * self.vdim].view(n, H, self.vdim)
            rate = torch.nn.functional.softplus(self.z[b].double() + self.dt_bias.double(), threshold=40).view(n, H, -1)
            decay = torch.exp(-torch.exp(self.a_log.double())[None, :, None] * rate)
            beta = torch.sigmoid(self.proj[b][:, 2:2 + H].double())
            S, o = torch.zeros_like(state[0]), []
            for t in range(n):
                S = S * decay[t][:, :, None]
                u = beta[t][:, None] * (v[t] - (S * k[t][:, :, None]).sum(1))
                S = S + k[t][:, :, None] * u[:, None]
                o.append((S * q[t][:, :, None]).sum(1))
            outs.append(torch.stack(o))
            state[int(self.slots[b])] = S
        return outs, state


# every size class of key channels, columns that do not fill a block or a pair, rings of six buffers that wrap
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("dim, vdim, pad", [(12, 20, 0), (16, 64, 0), (32, 33, 0), (48, 40, 1), (64, 64, 0), (96, 96, 0), (128, 128, 0),
                                            (128, 31, 4), (200, 40, 0), (256, 64, 0), (300, 35, 0)])
def test_delta_prompts_pieces_and_single_tokens(dim, vdim, pad, per_head, dtype):
    delta = Delta([47, 130, 1, 48], 4, 2, dim, vdim, dtype, per_head, pad)
    outs, state = delta.walk([])
    want, want_state = delta.exact()
    for got, exact in zip(outs + [state], want + [want_state]):
        assert (got.double() - exact).abs().max() <= 2e-5 * exact.abs().max()       # as for gated linear attention
    for cuts in ([3, 19, 20, 51, 52], list(range(1, 50)) + [80]):
        pieces, state1 = delta.walk(cuts)
        assert all(torch.equal(a, b) for a, b in zip(pieces, outs)) and torch.equal(state, state1)


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("dim, vdim, seqs", [(128, 128, 9), (64, 64, 40), (16, 32, 80), (96, 40, 64), (256, 64, 24)])
def test_delta_in_a_large_step_and_alone(dim, vdim, seqs, per_head):
    """Many sequences take two columns a lane (and other blocks), one alone may take one: the same bits."""
    delta = Delta([70, 9, 1, 33] + [5] * (seqs - 4), 8, 4, dim, vdim, torch.bfloat16, per_head)
    outs, state = delta.walk([])
    for b in (0, 1, 2, 3, seqs - 1):
        alone = delta.state()
        o, = delta.step(alone, [(b, 0, delta.lens[b])])
        assert torch.equal(o, outs[b]) and torch.equal(alone[delta.slots[b]], state[delta.slots[b]])
