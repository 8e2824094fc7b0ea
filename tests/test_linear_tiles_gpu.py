"""The float32 product's tiles (64 x 64 and 128 x 64, 96 and 128 outputs a block), each at its edges: against float64, and a row of a
large product bit for bit as the row alone, which takes another tile."""
import pytest
import torch

from rust_inference_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _close(got, x, w):
    """A chain of K multiply-adds: each rounds a sum of no more than the magnitudes' sum by 2^-24 of it."""
    want, most = x.double() @ w.double().transpose(-1, -2), x.double().abs() @ w.double().abs().transpose(-1, -2)
    assert ((got.double() - want).abs() <= x.shape[-1] * 2.0 ** -24 * most).all()


# whole groups of 16 k, whole 16-byte pieces but a rest of a group, no 16-byte pieces, less than a group
@pytest.mark.parametrize("K", [64, 100, 37, 5])
@pytest.mark.parametrize("M, N", [
    (1, 1), (64, 64), (65, 63), (3, 4097),              # 64 x 64
    (129, 4096), (200, 4001), (256, 4033),              # 128 x 64
    (65, 12288), (128, 12200), (300, 4093), (127, 11905),    # 128 x 96
    (512, 4096), (450, 4090), (511, 4000)])             # 128 x 128
def test_tiles_of_a_product(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x, w = torch.randn((M, K), generator=g, device=DEV), torch.randn((N, K), generator=g, device=DEV)
    got = ops.linear(x, w)
    _close(got, x, w)
    for row in (0, M // 2, M - 1):
        assert torch.equal(ops.linear(x[row:row + 1].contiguous(), w)[0], got[row])


@pytest.mark.parametrize("M, H, N, K", [(1, 3, 65, 20), (140, 32, 64, 36), (300, 32, 90, 21), (512, 32, 128, 40)])
def test_tiles_of_products_per_head(M, H, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x = torch.randn((M, H, K + 4), generator=g, device=DEV)[:, :, 4:]        # rows of a wider block
    w = torch.randn((H, N, K), generator=g, device=DEV)
    got = ops.linear_heads(x, w)
    for h in range(H):
        _close(got[:, h], x[:, h], w[h])
    assert torch.equal(ops.linear_heads(x[M - 1:], w)[0], got[M - 1])
