"""The kernels' dispatch rules on the GPU: calls on both sides of a rule give the same
results."""
import pytest

from spica_gb300 import GpuBVHAccel, scenes

pytestmark = pytest.mark.gpu


def _device_rays(n, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    org = torch.zeros((n, 4), device="cuda")
    dirs = torch.zeros((n, 4), device="cuda")
    org[:, :3] = 2.4 * torch.rand((n, 3), device="cuda", generator=g) - 1.2
    dirs[:, :3] = torch.randn((n, 3), device="cuda", generator=g)
    dirs[:, :3] /= dirs[:, :3].norm(dim=1, keepdim=True)
    dirs[:, 3] = 1.0e32
    return org, dirs


@pytest.mark.parametrize("levels", [4, 5])            # trees below and above 512 wide nodes
@pytest.mark.parametrize("rays", [(1 << 21) - 1, 1 << 21, (1 << 21) + 33])
def test_split_traversal_matches_whole_steps(gpulib, levels, rays):
    """Closest hits of 2^21 rays and more on larger trees are traced in the split form
    (the same order of triangle tests per ray), smaller batches in whole steps:
    every hit record is the same bit for bit."""
    import torch
    acc = GpuBVHAccel(scenes.displaced_sphere(levels=levels, seed=1)).construct()
    assert (acc.info().wide_nodes >= 512) == (levels == 5)
    org, dirs = _device_rays(rays, 7)
    out = torch.full((rays, 4), -1.0, device="cuda")
    acc.intersect_device(org, dirs, out)
    parts = torch.full((rays, 4), -1.0, device="cuda")
    for a in range(0, rays, 1 << 20):
        acc.intersect_device(org[a:a + (1 << 20)], dirs[a:a + (1 << 20)], parts[a:a + (1 << 20)])
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int32), parts.view(torch.int32))
    assert 0.1 < (out.view(torch.int32)[:, 1] >= 0).float().mean().item() < 1.0
