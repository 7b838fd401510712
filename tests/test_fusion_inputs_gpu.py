"""Device inputs of a fusion that the caller laid out in other ways than as tensors
of their own."""
import ctypes as C

import numpy as np
import pytest
import torch

from sensemap_b200 import _native as N
from sensemap_b200 import synthetic as syn
from sensemap_b200.fusion import FusionImage, FusionOptions, StereoFusion, fusion_structs

pytestmark = pytest.mark.gpu


def test_depth_maps_at_any_address():
    """Depth maps inside a byte buffer, at odd addresses."""
    scene = syn.planes_scene(seed=3, width=90, height=70, focal=72.0, num_src=3)
    images, overlaps = syn.fusion_inputs(scene, seed=1)
    device = [FusionImage(K=i.K, R=i.R, T=i.T, depth=torch.from_numpy(i.depth).cuda(),
                          normal=torch.from_numpy(i.normal).cuda(), color=torch.from_numpy(i.color).cuda())
              for i in images]
    options = FusionOptions()
    with StereoFusion(options, device, overlaps) as f:
        f.Run()
        want = f.GetFusedPoints().copy()
    assert len(want) > 20
    lib = N.lib()
    views, off, flat, memory, keep = fusion_structs(device, overlaps)
    for k, im in enumerate(images):
        buffer = torch.zeros(im.depth.nbytes + 16, dtype=torch.uint8, device="cuda")
        at = 1 + k % 3
        buffer[at:at + im.depth.nbytes] = torch.from_numpy(np.ascontiguousarray(im.depth).view(np.uint8).ravel()).cuda()
        keep.append(buffer)
        views[k].depth = buffer.data_ptr() + at
    torch.cuda.synchronize()
    h = C.c_void_p()
    N.check(lib.smvs_fusion_create(C.byref(options.to_c()), views, len(images), off.ctypes.data, flat.ctypes.data,
                                   memory, None, C.byref(h)))
    try:
        N.check(lib.smvs_fusion_run(h))
        n, nv = C.c_size_t(), C.c_size_t()
        N.check(lib.smvs_fusion_get_sizes(h, C.byref(n), C.byref(nv)))
        got = np.zeros(n.value, want.dtype)
        N.check(lib.smvs_fusion_get_points(h, got.ctypes.data, None, None))
    finally:
        lib.smvs_fusion_destroy(h)
    np.testing.assert_array_equal(got.view(np.uint8), want.view(np.uint8))
