"""Device inputs that are still being written when they are handed over, with no
stream given and with the default stream's handle, which is 0."""
import numpy as np
import pytest
import torch

from sensemap_b200.patch_match import PatchMatchACMMCuda, Problem, View
from sensemap_b200.pool import DepthMapPool
from tests.helpers import photometric_options, small_planes

pytestmark = pytest.mark.gpu

CYCLES = 400_000_000  # some 0.2 s of waiting on the GPU


def _late(array):
    """A tensor that holds zeros until torch's current stream gets to the values."""
    values = torch.from_numpy(np.ascontiguousarray(array)).float().cuda()
    out = torch.zeros_like(values)
    torch.cuda.synchronize()
    torch.cuda._sleep(CYCLES)
    out.copy_(values)
    return out


@pytest.mark.parametrize("stream", [None, 0])
def test_engine_and_pool_read_tensors_of_the_current_stream(stream):
    scene = small_planes(seed=3, w=96, h=72)
    opt = photometric_options(scene, iters=2)
    problem = Problem(0, [1, 2, 3, 4], [View(v.image, v.K, v.R, v.T) for v in scene.views])
    with PatchMatchACMMCuda(opt, problem) as pm:
        pm.Run()
        want = pm.GetDepthMap()
    late = [_late(v.image) for v in scene.views]
    views = [View(im, v.K, v.R, v.T) for im, v in zip(late, scene.views)]
    with PatchMatchACMMCuda(opt, Problem(0, [1, 2, 3, 4], views), stream=stream) as pm:
        pm.Run()
        np.testing.assert_array_equal(pm.GetDepthMap(), want)
    with DepthMapPool(max_active_jobs=1, image_storage=opt.image_storage, stream=stream) as pool:
        for i, v in enumerate(scene.views):
            pool.add_view(i, View(_late(v.image), v.K, v.R, v.T))
        job = pool.submit(opt, 0, [1, 2, 3, 4])
        pool.run_until_done([job])
        np.testing.assert_array_equal(pool.maps(job)["depth"], want)
