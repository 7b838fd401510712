"""The spread form of the checkerboard kernels (small launches: the warps of a
block share 32 pixels) against the thread-per-pixel form, which a persistent
launch always takes: the same maps bit for bit at sizes around its tiles of 32
columns x 2 rows, for the smallest and largest source counts, every window and
both passes; jobs with a prior keep the thread-per-pixel form."""
import numpy as np
import pytest

from sensemap_b200.patch_match import PatchMatchACMMCuda
from tests.helpers import perturbed_gt, photometric_options, problem_from_scene, small_planes

pytestmark = pytest.mark.gpu


def _maps(opt, problem, persistent):
    with PatchMatchACMMCuda(opt, problem) as pm:
        pm.SetTuning(32, True, 1, persistent)
        pm.Run()
        return pm.GetDepthMap(), pm.GetNormalMap(), pm.GetConfMap(), pm.GetCostMap(), pm.GetViewSelMap()


@pytest.mark.parametrize("size,sources,window,mode", [
    ((33, 17), 1, (5, 1), "photometric"), ((64, 32), 2, (3, 2), "photometric"), ((31, 33), 5, (5, 2), "photometric"),
    ((97, 65), 32, (5, 2), "photometric"), ((96, 64), 7, (7, 1), "photometric"), ((65, 48), 4, (3, 1), "geometric"),
    ((80, 47), 9, (4, 2), "geometric"), ((100, 61), 3, (7, 2), "geometric"), ((90, 51), 4, (5, 1), "prior"),
    ((66, 50), 4, (5, 2), "propagate")])
def test_spread_form_matches_thread_per_pixel(size, sources, window, mode):
    scene = small_planes(seed=11, w=size[0], h=size[1], f=0.8 * size[0], n_src=sources)
    given = mode != "photometric"
    depth = [v.depth_gt for v in scene.views] if given else None
    normal = [v.normal_gt for v in scene.views] if given else None
    problem = problem_from_scene(scene, depth_maps=depth, normal_maps=normal,
                                 init=perturbed_gt(scene) if given else None)
    opt = photometric_options(scene, iters=5, window_radius=window[0], window_step=window[1],
                              init_depth_random=not given, geom_consistency=mode == "geometric",
                              has_prior_depth=mode == "prior", propagate_depth=mode == "propagate")
    if mode == "prior":
        problem.prior_wgt = np.random.default_rng(3).random((size[1], size[0])).astype(np.float32)
    for a, b in zip(_maps(opt, problem, False), _maps(opt, problem, True)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("sources", [4, 10, 14, 20])
@pytest.mark.parametrize("window", [(3, 1), (5, 1), (7, 1), (3, 2), (4, 2), (5, 2), (7, 2)])
def test_every_instance_matches_thread_per_pixel(window, sources):
    """Every compiled window with every view bucket of the thread-per-pixel kernels
    (8, 12, 16, 32), photometric and geometric: each is an instance of its own,
    whose roundings the compiler could choose differently."""
    scene = small_planes(seed=11, w=100, h=75, f=80.0, n_src=sources)
    init = perturbed_gt(scene)
    for geometric in (False, True):
        problem = problem_from_scene(scene, depth_maps=[v.depth_gt for v in scene.views] if geometric else None,
                                     normal_maps=[v.normal_gt for v in scene.views] if geometric else None,
                                     init=init if geometric else None)
        opt = photometric_options(scene, iters=5, window_radius=window[0], window_step=window[1],
                                  init_depth_random=not geometric, geom_consistency=geometric)
        for a, b in zip(_maps(opt, problem, False), _maps(opt, problem, True)):
            np.testing.assert_array_equal(a, b)
