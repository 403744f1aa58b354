"""The fp8 SwiGLU feed-forward as one node: bit for bit the two fp8 Linear nodes around the SwiGLU kernel."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _mlp(dim, ffn, scale=0.05):
    from kempnerforge_b200.models.mlp import SwiGLUMLP
    from kempnerforge_b200.ops import fp8

    torch.manual_seed(0)
    with torch.device(DEV):
        mlp = SwiGLUMLP(dim, ffn).to(torch.bfloat16)
    with torch.no_grad():
        for p in mlp.parameters():
            p.normal_(0.0, scale)
    fp8.convert_model(mlp)
    return mlp


def _run(mlp, x, dy, need_x=True):
    mlp.zero_grad(set_to_none=True)
    xl = x.clone().requires_grad_(need_x)
    y = mlp(xl)
    y.backward(dy)
    return [y.detach(), xl.grad] + [p.grad for p in mlp.parameters()]


def _equal(a, b):
    return all((u is None and v is None) or torch.equal(u, v) for u, v in zip(a, b)) and len(a) == len(b)


@pytest.mark.parametrize("t,dim,ffn", [(16, 32, 16), (48, 64, 272), (400, 256, 1040), (2000, 1024, 3584)])
def test_equals_the_separate_nodes(native_lib, monkeypatch, t, dim, ffn):
    from kempnerforge_b200.ops import fp8

    mlp = _mlp(dim, ffn)
    x, dy = (torch.randn(t, dim, device=DEV).bfloat16() for _ in range(2))
    used, native = [], fp8.swiglu_mlp
    monkeypatch.setattr(fp8, "swiglu_mlp", lambda *a: used.append(native(*a)) or used[-1])
    got = _run(mlp, x, dy)
    zero = _run(mlp, torch.zeros_like(x), dy)
    for i, p in enumerate(mlp.parameters()):
        p.requires_grad_(i == 1)
    frozen = _run(mlp, x, dy, need_x=False)
    assert all(u is not None for u in used) and native_lib.read_status() == 0
    monkeypatch.setattr(fp8, "swiglu_mlp", lambda *a: None)
    assert _equal(frozen, _run(mlp, x, dy, need_x=False))
    for p in mlp.parameters():
        p.requires_grad_(True)
    assert _equal(got, _run(mlp, x, dy)) and _equal(zero, _run(mlp, torch.zeros_like(x), dy))


def test_second_backward_and_other_layers(native_lib):
    from kempnerforge_b200.ops import fp8

    mlp = _mlp(64, 128)
    x = torch.randn(3, 16, 64, device=DEV).bfloat16().requires_grad_(True)
    y = mlp(x)
    first = torch.autograd.grad(y.float().square().sum(), [x, *mlp.parameters()], retain_graph=True)
    assert _equal(first, torch.autograd.grad(y.float().square().sum(), [x, *mlp.parameters()]))
    w = [mlp.gate_proj.weight, mlp.up_proj.weight, mlp.down_proj.weight]
    assert fp8.swiglu_mlp(x[:, :5], *w) is None and fp8.swiglu_mlp(x.float(), *w) is None   # 15 rows; fp32
    assert fp8.swiglu_mlp(x, w[0], w[1], w[2].detach().clone()) is None                     # a weight that is not tagged
