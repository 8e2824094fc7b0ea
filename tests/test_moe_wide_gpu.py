"""The routed feed-forward of steps with many tokens: the tcgen05 grouped products (plain and with the gate in the epilogue, rows
gathered and scattered), the plan of wide tiles, the router by tiles of tokens and the combination, at the edges of their tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ops():
    from rust_inference_b200 import ops
    return ops


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _plan_rows(plan, experts):
    """(expert, pair) of every row of a plan's tiles, after a look at the plan itself."""
    perm, tiles, meta, bm = plan
    n, rows = meta.tolist()
    perm, tiles = perm.cpu().numpy(), tiles.cpu().numpy()[:n]
    assert (tiles[:, 2] > 0).all() and (tiles[:, 2] <= bm).all() and tiles[:, 2].sum() == rows
    at = 0
    for e, r0, k in tiles:
        assert r0 == at and 0 <= e < experts
        at += k
    return [(int(e), int(perm[r])) for e, r0, k in tiles for r in range(r0, r0 + k)]


@pytest.mark.parametrize("pairs, experts", [(1, 1), (127, 1), (256, 2), (257, 3), (1000, 16), (5000, 300)])
@pytest.mark.parametrize("wide", [False, True])
def test_plan_lists_every_pair_once(pairs, experts, wide):
    ops = _ops()
    idx = torch.randint(0, experts + 2, (pairs, 1), generator=_gen(pairs), device=DEV, dtype=torch.int32)
    idx[idx == 1] = 0                                            # an expert without pairs (where there is a second one)
    listed = _plan_rows(ops.moe_plan(idx, experts, wide), experts)
    chosen = idx.flatten().cpu().numpy()
    want = [(int(e), p) for p, e in enumerate(chosen) if e < experts]
    assert sorted(listed) == sorted(want) and [e for e, _ in listed] == sorted(e for e, _ in listed)


# a row's product is a float32 sum of K bfloat16 products: 2^-8 for the rounding of a bfloat16 result, and for the order of the
# sums some 1e-6 of the sum of magnitudes
@pytest.mark.parametrize("tokens, top, E, N, K", [(1, 1, 1, 8, 8), (129, 1, 2, 256, 64), (200, 3, 5, 264, 72), (77, 2, 3, 40, 128),
                                                  (300, 4, 4, 520, 200), (2100, 2, 7, 96, 1000), (640, 2, 3, 1376, 136),
                                                  (255, 1, 1, 255, 64), (257, 1, 1, 257, 448), (4000, 2, 2, 512, 128)])
@pytest.mark.parametrize("out_f32", [False, True])
def test_grouped_product_gathers_and_scatters(tokens, top, E, N, K, out_f32):
    ops = _ops()
    g = _gen(tokens * N + K)
    x = torch.randn((tokens, K), generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn((E, N, K), generator=g, device=DEV) * 0.1).to(torch.bfloat16)
    idx = torch.randint(0, E + 1, (tokens, top), generator=g, device=DEV, dtype=torch.int32)
    plan = ops.moe_plan(idx, E, True)
    rows = tokens * top
    flat = idx.flatten().long()
    live = flat < E
    token = torch.arange(rows, device=DEV) // top
    want = torch.zeros((rows, N), dtype=torch.float64, device=DEV)
    for e in range(E):
        at = (flat == e).nonzero().flatten()
        want[at] = x[token[at]].double() @ w[e].double().t()
    tol = 1e-5 if out_f32 else 2.0 ** -8
    bound = (x.double().abs().max() * w.double().abs().sum(-1).max()) * 1e-6
    dt = torch.float32 if out_f32 else None
    got = ops.moe_grouped_linear(x, w, plan, rows, gather_div=top, scatter=True, out_dtype=dt)
    assert ((got.double() - want)[live].abs() <= tol * want[live].abs() + bound).all()
    # rows as the plan lists them: gathered and left there, then read in place and scattered back
    perm = plan[0].long()[:int(live.sum())]
    listed = ops.moe_grouped_linear(x, w, plan, rows, gather_div=top, out_dtype=dt)
    assert torch.equal(listed[:len(perm)], got[perm])
    packed = torch.zeros((rows, K), dtype=torch.bfloat16, device=DEV)
    packed[:len(perm)] = x[token[perm]]
    back = ops.moe_grouped_linear(packed, w, plan, rows, scatter=True, out_dtype=dt)
    assert torch.equal(back[live], got[live])


@pytest.mark.parametrize("kind, limit, alpha", [("silu", 0.0, 1.0), ("gelu_tanh", 0.0, 1.0), ("clamped_swish", 1.5, 1.702)])
@pytest.mark.parametrize("tokens, top, E, N, K", [(130, 2, 3, 128, 64), (260, 3, 2, 132, 96), (90, 1, 4, 17, 40), (700, 2, 2, 352, 264)])
def test_gate_in_the_epilogue(kind, limit, alpha, tokens, top, E, N, K):
    ops = _ops()
    g = _gen(tokens + N)
    x = torch.randn((tokens, K), generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn((E, 2 * N, K), generator=g, device=DEV) * 0.2).to(torch.bfloat16)
    idx = torch.randint(0, E, (tokens, top), generator=g, device=DEV, dtype=torch.int32)
    plan = ops.moe_plan(idx, E, True)
    rows = tokens * top
    got = ops.moe_grouped_gated(x, w, plan, rows, kind, limit, alpha, gather_div=top)
    perm = plan[0].long()
    e = idx.flatten().long()[perm]
    both = torch.stack([x[perm // top].double() @ w[i].double().t() for i in range(E)])[e, torch.arange(rows, device=DEV)]
    gate, up = both[:, :N], both[:, N:]
    if kind == "silu":
        want = gate * torch.sigmoid(gate) * up
    elif kind == "gelu_tanh":
        want = torch.nn.functional.gelu(gate, approximate="tanh") * up
    else:
        gate, up = torch.clamp(gate, max=limit), torch.clamp(up, -limit, limit)
        want = gate * torch.sigmoid(alpha * gate) * (up + 1.0)
    scale = want.abs().max()
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * scale).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
# (the number of SMs, 148, is where the forms meet; widths whose last run of 512 k is four k and a whole one)
@pytest.mark.parametrize("tokens, D, N, top, rule", [(149, 516, 18, 4, {}), (150, 1028, 34, 3, {}), (200, 1024, 7, 2, {}), (256, 128, 4, 2, {}), (257, 132, 18, 4, {}), (300, 4096, 18, 4, {}), (512, 260, 33, 3, {}),
                                                     (391, 512, 16, 4, dict(score="sigmoid", groups=4, keep=2, scale=2.0, renormalize=False)),
                                                     (259, 640, 9, 3, dict(score="logits"))])
def test_router_by_tiles_gives_the_bits_of_a_block_per_token(tokens, D, N, top, rule, dtype):
    ops = _ops()
    g = _gen(tokens + D)
    x = torch.randn((tokens, D), generator=g, device=DEV).to(dtype)
    router = torch.randn((N, D), generator=g, device=DEV) * 0.1
    correction = None if rule.get("score") == "logits" else torch.randn((N,), generator=g, device=DEV) * 0.1
    bias = torch.randn((N,), generator=g, device=DEV) if rule.get("score") == "logits" else None
    idx, weight = ops.moe_route(x, router, correction, top, bias=bias, **rule)
    for lo in range(0, tokens, 100):                             # few tokens: a block per token
        hi = min(lo + 100, tokens)
        i1, w1 = ops.moe_route(x[lo:hi].clone(), router, correction, top, bias=bias, **rule)
        assert torch.equal(idx[lo:hi], i1) and torch.equal(weight[lo:hi], w1)


# up to 32 choices a lane keeps each; with more they go through memory
@pytest.mark.parametrize("top", [31, 32, 33, 70])
@pytest.mark.parametrize("tokens", [3, 300])
@pytest.mark.parametrize("score, renormalize", [("softmax", True), ("sigmoid", False), ("logits", True)])
def test_router_with_more_choices_than_lanes(tokens, top, score, renormalize):
    ops = _ops()
    g = _gen(top)
    D, N = 64, 100
    x = torch.randn((tokens, D), generator=g, device=DEV)
    router = torch.randn((N, D), generator=g, device=DEV) * 0.2
    correction = None if score == "logits" else torch.randn((N,), generator=g, device=DEV) * 0.1
    idx, weight = ops.moe_route(x, router, correction, top, score=score, scale=1.5, renormalize=renormalize)
    logits = x.double() @ router.double().t()
    scores = {"softmax": logits.softmax(-1), "sigmoid": logits.sigmoid(), "logits": logits}[score]
    choice = scores if correction is None else scores + correction.double()
    # the chosen are distinct, in descending order, and nothing that was left out is better (float32 sums of 64 products: 1e-5)
    assert (idx.sort(1).values.diff(dim=1) > 0).all()
    at = choice.gather(1, idx.long())
    left = choice.scatter(1, idx.long(), float("-inf")).max(1).values
    assert (at.diff(dim=1) <= 1e-5).all() and (left <= at[:, -1] + 1e-5).all()
    want = scores.gather(1, idx.long())
    want = want.softmax(-1) if score == "logits" else want / want.sum(-1, keepdim=True) if renormalize else want
    assert ((weight.double() - 1.5 * want).abs() <= 1e-5 * (1 + want.abs())).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens, D, top, extra", [(1, 4, 1, True), (5, 1028, 9, False), (600, 36, 4, True), (7, 30, 3, True), (513, 2048, 5, False)])
def test_combination_in_groups_of_four(tokens, D, top, extra, dtype):
    ops = _ops()
    g = _gen(D)
    E = 6
    pair = torch.randn((tokens * top, D), generator=g, device=DEV)
    idx = torch.randint(0, E + 2, (tokens, top), generator=g, device=DEV, dtype=torch.int32)
    weight = torch.rand((tokens, top), generator=g, device=DEV)
    x, more = (torch.randn((tokens, D), generator=g, device=DEV).to(dtype) for _ in range(2))
    for w in (weight, None):
        got = ops.moe_combine(pair, idx, w, x, E, more if extra else None)
        want = torch.zeros((tokens, D), dtype=torch.float64, device=DEV)
        for j in range(top):
            v = torch.where((idx[:, j] >= E)[:, None], x.double(), pair.view(tokens, top, D)[:, j].double())
            want += (w[:, j:j + 1].double() if w is not None else 1.0 / top) * v
        want = want + more.double() if extra else want
        tol = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-6
        assert ((got.double() - want).abs() <= tol * want.abs() + (top + 1) * 2.0 ** -22).all()


# tiles of 32 rows whose blocks need fewer rounds with three stages of the ring (16 x 43 blocks on 148 SMs), and one that has four; k in
# whole stages, with a rest, less than the ring
@pytest.mark.parametrize("E, N", [(16, 1376), (4, 64)])
@pytest.mark.parametrize("K", [256, 200, 72])
def test_few_tokens_in_rings_of_three_and_four_stages(E, N, K):
    ops = _ops()
    g = _gen(N + K)
    tokens, top = 24, 2
    x = torch.randn((tokens, K), generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn((E, 2 * N, K), generator=g, device=DEV) * 0.1).to(torch.bfloat16)
    idx = torch.randint(0, E, (tokens, top), generator=g, device=DEV, dtype=torch.int32)
    plan = ops.moe_plan(idx, E)
    e, rows = idx.flatten().long(), tokens * top
    want = torch.einsum("rk,rnk->rn", x.double().repeat_interleave(top, 0), w.double()[e])
    got = ops.moe_grouped_linear(x, w, plan, rows, gather_div=top, scatter=True, out_dtype=torch.float32)
    # float32 sums of K products, in any order: K 2^-24 of the magnitudes' sum
    most = torch.einsum("rk,rnk->rn", x.double().abs().repeat_interleave(top, 0), w.double().abs()[e])
    assert ((got.double() - want).abs() <= K * 2.0 ** -24 * most).all()
    gated = ops.moe_grouped_gated(x, w, plan, rows, "silu", gather_div=top)
    gate, up = want[plan[0].long()].chunk(2, dim=1)
    want = gate * torch.sigmoid(gate) * up
    assert ((gated.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * want.abs().max()).all()


def test_copying_warps_that_stop_at_different_stages():
    """The way out of a wait that has run out, with one copying warp of each block of the first pair of blocks stopped (by a test-only
    define, for K = 1536) before its fourth stage while the other copies go on to the end of the ring.  Error 5 is reported, what was
    started lands, the kernel returns, the other tiles are right, and so is the next launch.  Nothing hangs or faults: the waits are the
    bounded ones."""
    import os
    import subprocess
    import sys
    code = r'''
import time, torch
from rust_inference_b200 import ops
torch.manual_seed(0)
flag = ops.error_flag("cuda")
def run(K):
    x = torch.randn(700, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(2, 520, K, device="cuda") * 0.1).to(torch.bfloat16)
    idx = torch.randint(0, 2, (700, 1), device="cuda", dtype=torch.int32)
    plan = ops.moe_plan(idx, 2, True)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    y = ops.moe_grouped_linear(x, w, plan, 700, gather_div=1, out_dtype=torch.float32)
    torch.cuda.synchronize()
    ms = (time.perf_counter() - t0) * 1e3
    perm = plan[0].long()
    want = torch.stack([x[perm].float() @ w[e].float().t() for e in range(2)])[idx.flatten().long()[perm], torch.arange(700, device="cuda")]
    near = (y - want).abs() <= 1e-3 * want.abs().max()
    return near, ms
assert run(1024)[0].all() and int(flag.item()) == 0               # builds and loads the library (another K: nothing stops)
near, ms = run(1536)
assert int(flag.item()) == 5, int(flag.item())
flag.zero_()
assert near[256:].all() and near[:, 256:].all(), "the other tiles"
assert not near[:256, :256].all(), "nothing was stopped"
assert run(1536 + 64)[0].all() and int(flag.item()) == 0
print("gave up after %.1f ms" % ms)
'''
    env = dict(os.environ, RUST_INFERENCE_B200_DEFINES="MT_TEST_STOP_COPY_K=1536", PYTHONPATH=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600, env=env)
    assert r.returncode == 0, r.stdout + r.stderr
    # the products' wait and those of the epilogues (4 ms each, side by side); a copy that never landed would add one for each stage
    ms = float(r.stdout.split("after")[1].split()[0])
    assert 3.0 <= ms <= 2000.0, r.stdout
