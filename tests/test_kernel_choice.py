"""Which kernel an operation takes, looked at without a GPU: the launches are recorded instead of made."""
import pytest
import torch

from rust_inference_b200 import ops


@pytest.fixture
def launches(monkeypatch):
    """The (library, entry point, arguments) of every launch; tensors may lie on the CPU."""
    calls = []

    def need(t, name, dtype=None, shape=None):
        if not t.is_contiguous() or (dtype is not None and t.dtype != dtype) or (shape is not None and tuple(t.shape) != tuple(shape)):
            raise ops.KernelError(f"{name}: {t.dtype} {tuple(t.shape)}")

    monkeypatch.setattr(ops, "_need", need)
    monkeypatch.setattr(ops, "_call", lambda lib, fn, *args, **kw: calls.append((lib, fn, args)))
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "error_flag", lambda device: torch.zeros(1, dtype=torch.int32))
    return calls


def _plan(pairs, experts, rows):
    """What ``moe_plan`` returns for tiles of ``rows`` rows (the numbers in it do not matter here)."""
    return torch.zeros(pairs, dtype=torch.int32), torch.zeros((1 + experts, 3), dtype=torch.int32), torch.zeros(2, dtype=torch.int32), rows


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("gather", [0, 2])
def test_plans_of_wide_tiles_are_for_bfloat16(launches, dtype, gather):
    a, w = torch.zeros((4, 16), dtype=dtype), torch.zeros((3, 24, 16), dtype=dtype)
    plan = _plan(8, 3, ops.MOE_TILE_ROWS_WIDE)
    with pytest.raises(ops.KernelError):
        ops.moe_grouped_linear(a, w, plan, 8, gather_div=gather)
    with pytest.raises(ops.KernelError):
        ops.moe_grouped_gated(a, w, plan, 8, "silu", gather_div=gather)
    assert launches == []
    a, w = a.bfloat16(), w.bfloat16()
    ops.moe_grouped_linear(a, w, plan, 8, gather_div=gather)
    ops.moe_grouped_gated(a, w, plan, 8, "silu", gather_div=gather)
    assert [fn for _, fn, _ in launches] == (["ri_moe_gather"] if gather else []) + ["ri_moe_tc"] + (["ri_moe_gather"] if gather else []) + ["ri_moe_tc"]
