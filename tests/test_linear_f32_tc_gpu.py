"""The float32 product on the tensor cores: sizes at the edges of its tiles, stages and launches against float64, a row of a large
product bit for bit as the row alone, and values that are not finite."""
import pytest
import torch

from rust_inference_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    return torch.randn((M, K), generator=g, device=DEV), torch.randn((N, K), generator=g, device=DEV)


def _close(got, x, w):
    """What is left out of a product is below 2^-24 of it, the two additions of 16 products of 16 bits cut a sum of 32 k off by 2^-23 of its
    magnitudes each, the small terms' sum (2^-7 of the magnitudes at most) is cut off ten times a stage by 2^-23, and the
    K / 32 + 1 additions of sums round by 2^-24 each."""
    want, most = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert ((got.double() - want).abs() <= (x.shape[1] / 32 + 32) * 2.0 ** -24 * most).all()


def _multiply_adds(x, w):
    y = torch.empty((x.shape[0], w.shape[0]), device=DEV)
    ops._call("linear_f32", "ri_linear_f32", x.data_ptr(), w.data_ptr(), y.data_ptr(), x.shape[0], w.shape[0], x.shape[1], ops._stream())
    return y


# one to three rounds of the rings, a last stage of 4 and of 28 k
@pytest.mark.parametrize("K", [128, 132, 412, 1056])
@pytest.mark.parametrize("M, N", [
    (1, 1), (16, 128), (17, 129), (64, 4096), (65, 700),        # up to 64 tokens a block
    (80, 9500), (128, 9473), (250, 4000),                       # up to 128
    (176, 9473), (512, 6144), (353, 6100)])                     # up to 176
def test_sizes(M, N, K):
    x, w = _inputs(M, N, K)
    assert ops._takes_f32_tc(K, w.data_ptr())
    got = ops.linear(x, w)
    _close(got, x, w)
    for row in (0, M // 2, M - 1):
        assert torch.equal(ops.linear(x[row:row + 1].contiguous(), w)[0], got[row])
    assert torch.equal(ops.linear(x, w), got)


def test_no_larger_error_than_multiply_adds():
    for M, N, K in ((40, 300, 128), (300, 4000, 128), (100, 500, 1000), (300, 1000, 4096)):
        x, w = _inputs(M, N, K)
        want = x.double() @ w.double().T
        errors = [((y.double() - want).norm() / want.norm()).item() for y in (ops.linear(x, w), _multiply_adds(x, w))]
        assert errors[0] <= errors[1], (K, errors)


def _sparse(M, K, entries):
    x, g = torch.randn((M, K), device=DEV), torch.Generator(device=DEV).manual_seed(entries)
    return x * torch.zeros_like(x).scatter_(1, torch.rand((M, K), generator=g, device=DEV).topk(entries, 1).indices, 1.0)


@pytest.mark.parametrize("K", [128, 4096])
@pytest.mark.parametrize("M", [60, 120, 700])                     # the three variants of the kernel
def test_sums_with_few_terms_and_of_one_sign(M, K):
    w = torch.randn((9473, K), generator=torch.Generator(device=DEV).manual_seed(K), device=DEV)
    # one product: its rounding to float32, 2^-24, and what is left out of it, below 2^-24.1
    x = _sparse(M, K, 1)
    want = x.double() @ w.double().T
    assert ((ops.linear(x, w).double() - want).abs() <= 1.95 * 2.0 ** -24 * want.abs()).all()
    near = 1 + 2.0 ** -7 + 1e-3 * torch.rand((M, K), device=DEV)       # values whose middle parts are large
    for x, w in [(_sparse(M, K, n), w) for n in (2, 4, 8, 32)] + [(near, 1 + 2.0 ** -7 - 2.0 ** -23 + 1e-4 * w.abs())]:
        want = x.double() @ w.double().T
        errors = [(y.double() - want).norm().item() for y in (ops.linear(x, w), _multiply_adds(x, w))]
        assert errors[0] <= errors[1], errors


# float32 numbers whose third parts are below bfloat16's smallest, in either operand; sums that are below float32's smallest normal number
@pytest.mark.parametrize("scale_x, scale_w", [(1e-34, 1.0), (1e-37, 1.0), (1.0, 1e-36), (1e5, 1e-40), (1e-42, 1e5), (1e-20, 1e-16)])
def test_small_values(scale_x, scale_w):
    x, w = _inputs(70, 300, 256)
    x, w = x * scale_x, w * scale_w
    want, most = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    got, multiply_adds = ops.linear(x, w), _multiply_adds(x, w)
    assert ((got.double() - want).abs() <= 8 * 2.0 ** -24 * most + 2.0 ** -150).all()
    assert (got.double() - want).norm() <= (multiply_adds.double() - want).norm()


def test_values_beyond_the_scaled_range_are_taken_by_multiply_adds():
    x, w = _inputs(70, 300, 256)
    for a, b in ((x * 1e35, w * 1e-3), (x * 1e-3, w * 1e35), (x * 1e15, w * 1e15)):          # 2^112 for a value, 2^96 for a sum
        got, want = ops.linear(a, b), _multiply_adds(a, b)
        far = want.abs() > 2.0 ** 97
        assert torch.isfinite(want).all() and far.any() and torch.equal(got[far], want[far])
        _close(got, a, b)


def test_tokens_a_block_stay_below_the_largest_variant():
    """Where the largest variant cannot be taken (its warps hand registers over, which the compiler has to have given them) the rule stays
    at 128 tokens a block."""
    tokens = lambda rows, N, most: ops._fn("linear_f32", "ri_linear_f32_tc_tokens")[0](rows, N, 148, most)
    assert tokens(512, 6144, 176) == 176
    assert all(tokens(rows, N, 128) <= 128 for rows in (1, 100, 176, 512, 3000) for N in (1, 6144, 9473))


def test_a_wait_that_runs_out():
    """Built with a test-only define, the first block of a launch with K = 1536 leaves out a copy of W.  Error 5 is reported, the kernel
    returns, the other blocks' outputs are right, and so is the next launch.  Nothing hangs or faults: the waits are the bounded ones."""
    import os
    import subprocess
    import sys
    code = r'''
import time, torch
from rust_inference_b200 import ops
torch.manual_seed(0)
flag = ops.error_flag("cuda")
def run(M, K, N=9473):
    x, w = torch.randn(M, K, device="cuda"), torch.randn(N, K, device="cuda")
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    y = ops.linear(x, w)
    torch.cuda.synchronize()
    ms = (time.perf_counter() - t0) * 1e3
    want = x.double() @ w.double().t()
    return (y.double() - want).abs() <= 1e-3, ms
for M in (40, 120, 176):                                          # the three variants
    assert run(M, 1024)[0].all() and int(flag.item()) == 0        # (another K: nothing is left out)
    near, ms = run(M, 1536)
    assert int(flag.item()) == 5, int(flag.item())
    flag.zero_()
    assert near[:, 128:].all() and not near.all(), "the other blocks"
    assert run(M, 2048)[0].all() and int(flag.item()) == 0
    print("gave up after %.1f ms" % ms)
'''
    env = dict(os.environ, RUST_INFERENCE_B200_DEFINES="LF_TEST_DROP_COPY_K=1536", PYTHONPATH=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600, env=env)
    assert r.returncode == 0, r.stdout + r.stderr
    for line in r.stdout.strip().splitlines():
        assert 3.0 <= float(line.split("after")[1].split()[0]) <= 2000.0, r.stdout


def test_rows_in_several_launches(monkeypatch):
    x, w = _inputs(2500, 200, 288)
    whole = ops.linear(x, w)
    monkeypatch.setattr(ops, "F32_TC_SCRATCH", 1)                # 1,024 rows a launch
    assert torch.equal(ops.linear(x, w), whole)


def test_rows_that_are_not_whole_pieces_take_multiply_adds():
    for K in (257, 258):
        x, w = _inputs(5, 70, K)
        assert not ops._takes_f32_tc(K, w.data_ptr()) and torch.equal(ops.linear(x, w), _multiply_adds(x, w))
    buffer = torch.randn(70 * 256 + 1, device=DEV)
    w = buffer[1:].view(70, 256)                                 # rows that do not start on 16 bytes
    x = torch.randn((5, 256), device=DEV)
    assert torch.equal(ops.linear(x, w), _multiply_adds(x, w))


def test_values_that_are_not_finite():
    x, w = _inputs(40, 200, 512)
    x[3, 7], x[5, 9], w[10, 100], x[21, 0] = float("inf"), float("nan"), float("-inf"), float("-inf")
    x[8, 20], w[20, 20] = 3.4e38, 3e38                           # a product that overflows
    # sums near the end of the range that stay inside it (512 products of 1e36: some 2e37, at most 2e38 on their way; a sum that
    # leaves the range for less than 32 k and returns is finite here and infinite as a chain)
    x[30] *= 1e36
    got, want = ops.linear(x, w), _multiply_adds(x, w)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    endless = torch.isinf(want)
    assert torch.equal(torch.isinf(got), endless) and torch.equal(got[endless], want[endless])
    near = torch.isfinite(want)
    assert ((got - want)[near].abs() <= 512 * 2.0 ** -23 * (x.abs().nan_to_num(posinf=0) @ w.abs().nan_to_num(posinf=0).T)[near]).all()


def test_replayed_from_a_graph():
    x, w = _inputs(7, 300, 512)
    want = ops.linear(x, w)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = ops.linear(x, w)
    x.copy_(x.flip(0))
    graph.replay()
    assert torch.equal(got, want.flip(0))
