"""The fused head and loss under the gradients it can be handed: one, another scalar, and the weight gradient of a kept graph
(repeated passes and flat gradient slots: test_kept_graphs_gpu.py)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(t=300, v=1000, d=128):
    g = torch.Generator(device="cuda").manual_seed(0)
    h = torch.randn(t, d, device="cuda", generator=g).bfloat16().requires_grad_(True)
    w = (torch.randn(v, d, device="cuda", generator=g) * 0.05).bfloat16().requires_grad_(True)
    lab = torch.randint(0, v, (t,), device="cuda", generator=g)
    lab[::7] = -100
    return h, w, lab


@pytest.mark.parametrize("factor", [1.0, 0.37, -2.0, 0.0])
def test_upstream_factor_and_kept_graphs(native_lib, factor):
    from kempnerforge_b200.ops import functional as F

    h, w, lab = _case()
    one = torch.autograd.grad(F.linear_cross_entropy(h, w, lab, 1e-3), [h, w])
    f = torch.tensor(factor).bfloat16()
    # in place (graph released) and out of place (kept): bf16 products of the same values
    want = [(a.float() * float(f)).bfloat16() for a in one]
    for a, b in zip(torch.autograd.grad(F.linear_cross_entropy(h, w, lab, 1e-3) * factor, [h, w]), want):
        assert torch.equal(a, b)
    loss = F.linear_cross_entropy(h, w, lab, 1e-3) * factor
    kept = torch.autograd.grad(loss, [w], retain_graph=True)[0].clone()
    assert torch.equal(kept, want[1])


@pytest.mark.parametrize("n", [1, 7, 8, 2049, 1 << 20])
@pytest.mark.parametrize("factor", [1.0, 0.25, float("inf"), float("nan")])
def test_scale_in_place(native_lib, n, factor):
    x = torch.randn(n, device="cuda").bfloat16()
    want = x * torch.tensor(factor, dtype=torch.bfloat16, device="cuda")
    native_lib.scale_(x, torch.tensor([factor], device="cuda"))
    assert torch.equal(torch.nan_to_num(x.float(), 9.0, 8.0, 7.0), torch.nan_to_num(want.float(), 9.0, 8.0, 7.0))
