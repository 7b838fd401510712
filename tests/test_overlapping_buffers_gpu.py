"""Device calls whose outputs lie over an input that they have read before: the same
maps as with buffers of their own."""
import pytest
import torch

from sensemap_b200 import _native as N
from sensemap_b200 import pyramid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1200, 800), (300, 200)])
def test_normals_resampled_over_the_depth_map(size):
    w, h = 600, 400
    gen = torch.Generator("cuda").manual_seed(1)
    depth = torch.rand(h, w, device="cuda", generator=gen)
    normal = torch.rand(3, h, w, device="cuda", generator=gen) - 0.5
    want_d, want_n = pyramid.resample_maps(depth, normal, *size)
    torch.cuda.synchronize()
    for at in (0, size[0] * size[1]):  # where the depth map starts among the normals
        buffer = torch.zeros(max(3 * size[0] * size[1], at + w * h), device="cuda")
        buffer[at:at + w * h] = depth.flatten()
        out = torch.empty_like(want_d)
        torch.cuda.synchronize()
        N.check(N.lib().smvs_resample_maps(buffer.data_ptr() + 4 * at, normal.data_ptr(), w, h, out.data_ptr(),
                                           buffer.data_ptr(), *size, None))
        torch.cuda.synchronize()
        assert torch.equal(out, want_d)
        assert torch.equal(buffer[:3 * size[0] * size[1]].view_as(want_n), want_n)
