"""The fp8 copies of weights that are kept between calls: they follow the native optimizers, and stay on their stream and out of graphs."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _mlp(flat):
    from kempnerforge_b200.models.mlp import SwiGLUMLP
    from kempnerforge_b200.parallel.flat import FlatParamGroup

    torch.manual_seed(3)
    mlp = SwiGLUMLP(256, 512).to(DEV, torch.bfloat16)
    for p in mlp.parameters():
        p._kf_fp8 = True
    return mlp, FlatParamGroup("unit", mlp.named_parameters()) if flat else None


def _weights(mlp):
    return [(mlp.gate_proj.weight, mlp.up_proj.weight), (mlp.down_proj.weight,)]


def _same(weights):
    """The copies that a call would use now are those of the weights as they are now."""
    from kempnerforge_b200.ops import fp8

    kept = fp8.quantized_weight(weights, want_t=True)
    fresh = fp8.quantize(torch.cat([w.detach() for w in weights]), want_t=True)
    return all(torch.equal(a, b) for a, b in zip(kept, fresh))


@pytest.mark.parametrize("how", ["adamw", "lion", "schedule free"])
def test_copies_follow_the_native_optimizers(native_lib, how):
    from kempnerforge_b200.training import optimizer as o

    mlp, fg = _mlp(how == "adamw")
    make = {"adamw": o.FusedAdamW, "lion": o.Lion, "schedule free": o.ScheduleFreeAdamW}[how]
    opt = make(mlp.parameters(), lr=0.05)
    if fg is not None:
        opt.attach_flat_groups([fg])
    x = torch.randn(256, 256, device=DEV).bfloat16()
    for _ in range(3):
        mlp(x).float().square().mean().backward()
        if fg is not None:
            fg.finalize_grads()
        before = native_lib.LAUNCH_COUNT
        opt.step()
        assert native_lib.LAUNCH_COUNT > before   # our kernels wrote the weights
        assert all(map(_same, _weights(mlp)))
        opt.zero_grad()
        if fg is not None:
            fg.zero_grad()
    assert native_lib.read_status() == 0


def test_a_captured_call_reads_the_weights_at_every_replay(native_lib):
    mlp, _ = _mlp(False)
    x = torch.randn(256, 256, device=DEV).bfloat16()
    with torch.no_grad():
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            mlp(x)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = mlp(x)
        assert all(map(_same, _weights(mlp)))     # nothing of the graph's memory is kept
        for p in mlp.parameters():
            p.mul_(-2)
        graph.replay()
        assert torch.equal(y, mlp(x)) and native_lib.read_status() == 0
    del graph


def test_copies_belong_to_the_stream_that_made_them(native_lib):
    from kempnerforge_b200.ops import fp8

    weights = _weights(_mlp(False)[0])[0]
    here = fp8.quantized_weight(weights, want_t=True)
    assert fp8.quantized_weight(weights, want_t=True)[1] is here[1]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        there = fp8.quantized_weight(weights, want_t=True)
    torch.cuda.current_stream().wait_stream(side)
    assert there[1] is not here[1] and all(torch.equal(a, b) for a, b in zip(here, there))


@pytest.mark.parametrize("how", ["lion", "schedule free"])
def test_a_kept_graph_still_runs_after_a_native_update(native_lib, how):
    """A second backward pass reads the weights as they are then, as before their writes were counted."""
    from kempnerforge_b200.training import optimizer as o

    torch.manual_seed(5)
    lin = torch.nn.Linear(256, 128, bias=False, device=DEV, dtype=torch.bfloat16)
    from kempnerforge_b200.ops import functional as F

    x = torch.randn(64, 256, device=DEV).bfloat16().requires_grad_(True)
    y = F.linear(x, lin.weight)
    y.sum().backward(retain_graph=True)
    {"lion": o.Lion, "schedule free": o.ScheduleFreeAdamW}[how](lin.parameters(), lr=0.5).step()
    x.grad = None
    y.sum().backward()
    assert torch.allclose(x.grad.float(), lin.weight.detach().float().sum(0).expand(64, -1), rtol=2**-7, atol=2**-5)
