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
    assert [fn for _, fn, _ in launches] == ["ri_moe_tc", "ri_moe_tc"]
    assert all((sent[0] is not None) == (gather > 0) and sent[2] == gather for _, _, sent in launches)


# latent rows (keys of 256 elements whose first ones are the values): what the tcgen05 kernel does not do stays with the mma.sync kernel
TCGEN05, MMA = "ri_attention_latent_tc", "ri_attention_prefill"


@pytest.mark.parametrize("form, want", [
    ({}, TCGEN05), (dict(window=40), TCGEN05), (dict(chunk=64), TCGEN05), (dict(keep=3), TCGEN05), (dict(v_dims=190), TCGEN05),
    (dict(max_new=64), TCGEN05),                                     # an upper bound of what a sequence brings
    (dict(chunk=64, keep=3), TCGEN05),                               # kept keys count beside a window only
    (dict(window=40, keep=3), MMA), (dict(keep=-1), MMA),
    (dict(scale=0.0), MMA), (dict(scale=-0.1), MMA), (dict(scale=1e-38), MMA), (dict(scale=float("nan")), MMA),
    (dict(v_dims=0), MMA), (dict(v_dims=256), MMA), (dict(softcap=20.0), MMA)])
def test_forms_of_latent_prompts(launches, monkeypatch, form, want):
    monkeypatch.setattr(ops, "_NO_TCGEN05", False)
    q, pool = torch.zeros((5, 2, 256), dtype=torch.bfloat16), torch.zeros((2, 1, 32, 256), dtype=torch.bfloat16)
    one = torch.zeros(1, dtype=torch.int32)
    args = {**dict(max_new=5, scale=0.1, window=0, v_dims=192), **form}
    ops.attention_prefill(q, pool, pool, torch.zeros((1, 1), dtype=torch.int32), one, torch.zeros(2, dtype=torch.int32), one, **args)
    (_, fn, sent), = launches
    assert fn == want
    if want == TCGEN05:
        assert sent[7] == 5 and sent[9] == 5                        # tokens; the most of one sequence is no more than that


@pytest.mark.parametrize("switch", [False, True])
def test_the_switch_leaves_the_routed_products_to_mma_sync(launches, monkeypatch, switch):
    from rust_inference_b200.config.specs import GatedFFSpec, MoESpec
    from rust_inference_b200.parts import BuildEnv, build_part, part_class
    monkeypatch.setattr(ops, "_NO_TCGEN05", switch)
    spec = MoESpec(hidden_size=16, experts=2, top=1, expert=GatedFFSpec(16, 24, gate="silu"))
    part = build_part("ffn", spec, BuildEnv(torch.bfloat16, torch.device("cpu")))
    infos = part_class("ffn", spec).param_infos(spec)
    part.load({n: torch.zeros(i.shape, dtype=torch.bfloat16 if i.role == "matrix" else torch.float32) for n, i in infos.items()})
    asked = []
    monkeypatch.setattr(ops, "moe_plan", lambda idx, experts, wide=False: asked.append(wide) or _plan(200, 2, 256 if wide else 32))
    part(torch.zeros((200, 16), dtype=torch.bfloat16), None)
    assert asked == [not switch]
    assert [fn for _, fn, _ in launches if fn.startswith(("ri_moe_tc", "ri_moe_grouped"))] == (
        ["ri_moe_grouped_gated", "ri_moe_grouped_linear"] if switch else ["ri_moe_tc", "ri_moe_tc"])
