"""Device inputs that are still being written when they are handed over: another
engine's maps, and tensors of torch's current stream, with no stream given and with
the default stream's handle, which is 0."""
import numpy as np
import pytest
import torch

from sensemap_b200 import synthetic as syn
from sensemap_b200.patch_match import PatchMatchACMMCuda, Problem, View
from sensemap_b200.pool import DepthMapPool
from sensemap_b200.pyramid import PyramidPatchMatch
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
def test_engine_reads_another_engines_unfinished_maps(stream):
    scene = syn.heightfield_scene(seed=0, width=800, height=600, num_src=4, device="cuda")
    images = [torch.from_numpy(np.ascontiguousarray(v.image)).float().cuda() for v in scene.views]
    src = [1, 2, 3, 4]

    def geometric(wait):
        views = [View(im, v.K, v.R, v.T) for im, v in zip(images, scene.views)]
        photo = []
        for r in range(5):
            opt = photometric_options(scene, iters=4, random_seed=r)
            pm = PatchMatchACMMCuda(opt, Problem(r, [i for i in range(5) if i != r], views), stream=stream)
            pm.Run()
            photo.append(pm)
        if wait:
            torch.cuda.synchronize()
        maps = [pm.DeviceDepthNormal() for pm in photo]
        views = [View(im, v.K, v.R, v.T, depth=m[0], normal=m[1]) for im, v, m in zip(images, scene.views, maps)]
        opt = photometric_options(scene, iters=2, geom_consistency=True, init_depth_random=False, random_seed=9)
        with PatchMatchACMMCuda(opt, Problem(0, src, views), stream=stream) as pm:
            pm.Run()
            out = pm.GetDepthMap(), pm.GetCostMap()
        for pm in photo:
            pm.close()
        return out

    for a, b in zip(geometric(False), geometric(True)):
        np.testing.assert_array_equal(a, b)


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


def test_pyramid_without_a_stream_equals_one_on_a_stream():
    scene = syn.heightfield_scene(seed=0, width=640, height=480, num_src=4, device="cuda")
    views = [View(torch.from_numpy(np.ascontiguousarray(v.image)).float().cuda(), v.K, v.R, v.T) for v in scene.views]
    problems = [(r, [i for i in range(5) if i != r]) for r in range(5)]
    opt = photometric_options(scene, iters=4)
    torch.cuda.synchronize()
    own = PyramidPatchMatch(opt, views, problems, levels=2, refine=[0]).Run()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ordered = PyramidPatchMatch(opt, views, problems, levels=2, refine=[0], stream=stream.cuda_stream).Run()
    torch.cuda.synchronize()
    assert torch.equal(own.depth[0], ordered.depth[0]) and torch.equal(own.normal[0], ordered.normal[0])
