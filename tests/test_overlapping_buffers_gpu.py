"""Device calls whose outputs lie over an input that they have read before: the same
maps as with buffers of their own."""
import ctypes as C

import numpy as np
import pytest
import torch

from sensemap_b200 import _native as N
from sensemap_b200 import init_maps as IM
from sensemap_b200 import pyramid
from tests.helpers import small_planes

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


def test_dense_points_under_the_maps():
    """Positions where the depth map goes, normals where the normal map goes."""
    w, h, n = 640, 480, 100000
    v = small_planes(w=32, h=24).views[0]
    K = np.array([[500.0, 0, 320], [0, 500, 240], [0, 0, 1]])
    gen = torch.Generator("cuda").manual_seed(2)
    camera = torch.rand(n, 3, device="cuda", generator=gen) * torch.tensor([3.0, 2.2, 3.0], device="cuda")
    camera += torch.tensor([-1.5, -1.1, 3.0], device="cuda")
    R = torch.tensor(np.asarray(v.R), dtype=torch.float32, device="cuda")
    T = torch.tensor(np.asarray(v.T), dtype=torch.float32, device="cuda")
    xyz = ((camera - T) @ R).contiguous()
    normals = (-(camera / camera.norm(dim=1, keepdim=True)) @ R).contiguous()
    want_d, want_n, _ = IM.init_depth_from_dense_points(w, h, K, v.R, v.T, xyz, normals)
    assert (want_d > 0).sum() > 10000
    assert 3 * n < w * h
    depth, normal = torch.zeros(w * h, device="cuda"), torch.zeros(3 * w * h, device="cuda")
    depth[:3 * n], normal[1000:1000 + 3 * n] = xyz.flatten(), normals.flatten()
    torch.cuda.synchronize()
    view = IM._view(w, h, K, v.R, v.T)
    N.check(N.lib().smvs_init_depth_from_dense_points(
        C.byref(view), depth.data_ptr(), normal.data_ptr() + 4000, n, IM.PLY_INIT_DEPTH_LEVEL, N.MEM_DEVICE,
        depth.data_ptr(), normal.data_ptr(), None, None))
    torch.cuda.synchronize()
    assert torch.equal(depth.view(h, w), want_d) and torch.equal(normal.view(3, h, w), want_n)
