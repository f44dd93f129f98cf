"""Gate and norm in groups of 128 to 1,023 columns, four a lane and load, and the widths around them: against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("group", [96, 124, 128, 132, 256, 260, 388, 512, 516, 528, 532, 600, 640, 704, 768, 800, 896, 900, 916, 1020, 1024])
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("types", [(torch.float32, torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32, torch.float32)])
@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("offset", [0, 1])
def test_gated_norm_by_group_width(group, mode, types, norm, offset):
    """Column slices of wider rows; `offset` 1 starts them off the four-value boundary, which the general kernel takes."""
    from picolm_b200 import ops
    torch.manual_seed(group + mode)
    T, C = 7, 3 * group
    x = torch.randn(T, C + 8, device=DEV).to(types[0])[:, offset:offset + C]
    gate = torch.randn(T, C + 8, device=DEV).to(types[1])[:, offset:offset + C] if mode else None
    w = torch.rand(group, device=DEV) + 0.5
    got = ops.gated_norm(x, types[2], weight=w if norm else None, eps=1e-5, group=group, weight_per_group=True, gate=gate, gate_mode=mode, norm=norm)
    z = x.double()
    ga = torch.nn.functional.silu(gate.double()) if mode else 1.0
    z = z * ga if mode == 1 else z
    if norm:
        z = (z.view(T, 3, group) * torch.rsqrt((z.view(T, 3, group) ** 2).mean(-1, keepdim=True) + 1e-5) * w.double()).view(T, C)
    z = z * ga if mode == 2 else z
    tol = dict(atol=1e-5, rtol=1e-5) if types[2] == torch.float32 else dict(atol=1e-3, rtol=2.0 ** -8)
    assert torch.allclose(got.double(), z, **tol)
