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
