"""Pools and engines in either form of the checkerboard kernels (a thread per
pixel, or a pixel spread over a block's warps), whatever the size of the launch
would choose: the same maps bit for bit, also while a pool's group grows and
shrinks across the line between the two."""
import contextlib

import numpy as np
import pytest

from sensemap_b200 import _native as N
from sensemap_b200.patch_match import PatchMatchACMMCuda
from sensemap_b200.pool import DepthMapPool
from tests.helpers import photometric_options, problem_from_scene, small_planes
from tests.test_pool_gpu import add_scene, assert_same, engine_maps, scenes  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu

RULE, SPREAD, PIXEL = 0, 1, 2


@contextlib.contextmanager
def _form(form):
    N.check(N.lib().smvs_test_sweep_form(form))
    try:
        yield
    finally:
        N.check(N.lib().smvs_test_sweep_form(RULE))


@pytest.mark.parametrize("form,tma", [(SPREAD, True), (PIXEL, True), (PIXEL, False)])
def test_pool_in_one_form_equals_engines_in_the_other(scenes, form, tma):  # noqa: F811
    """Jobs of two sizes, 3 and 4 sources and 4 to 6 iterations, one of them admitted
    while others run."""
    jobs = []
    with DepthMapPool(max_active_jobs=8, ref_tile_tma=tma) as pool, _form(form):
        for si, sc in enumerate(scenes):
            add_scene(pool, sc, 100 * si)
        for si, sc in enumerate(scenes):
            for r in (0, 1):
                opt = photometric_options(sc, iters=4 + r + si, random_seed=10 * si + r)
                srcs = [100 * si + i for i in range(len(sc.views)) if i != r]
                jobs.append((pool.submit(opt, 100 * si + r, srcs), sc, r, opt))
            pool.step()
        pool.run_until_done([j[0] for j in jobs])
        maps = [pool.maps(j[0]) for j in jobs]
    with _form(PIXEL if form == SPREAD else SPREAD):
        for got, (_, sc, r, opt) in zip(maps, jobs):
            assert_same(got, engine_maps(opt, problem_from_scene(sc, ref=r)))


@pytest.mark.parametrize("form", [SPREAD, PIXEL])
def test_geometric_pass_of_a_pool_in_either_form(scenes, form):  # noqa: F811
    sc = scenes[0]
    n = len(sc.views)
    srcs = [j for j in range(n) if j != sc.ref_index]
    opt = photometric_options(sc, iters=5, geom_consistency=True, init_depth_random=False, random_seed=77)
    depth, normal = [v.depth_gt for v in sc.views], [v.normal_gt for v in sc.views]
    with DepthMapPool(max_active_jobs=4) as pool, _form(form):
        add_scene(pool, sc, 0)
        for i in range(n):
            pool.set_view_maps(i, depth[i], normal[i])
        job = pool.submit(opt, sc.ref_index, srcs)
        pool.run_until_done([job])
        got = pool.maps(job)
    with _form(PIXEL if form == SPREAD else SPREAD):
        prob = problem_from_scene(sc, depth_maps=depth, normal_maps=normal,
                                  init=(depth[sc.ref_index], normal[sc.ref_index]))
        assert_same(got, engine_maps(opt, prob))


@pytest.mark.parametrize("use_graphs", [True, False])
def test_group_that_crosses_the_line_and_comes_back(use_graphs):
    """Radius 3, step 2, 4 sources: up to 10,000 pixels a colour are spread. One job
    of 160x120 has 9,600; two more join it for some of its steps."""
    sc = small_planes(seed=41)
    opts = [photometric_options(sc, iters=it, window_radius=3, window_step=2, random_seed=20 + r)
            for r, it in enumerate((9, 3, 4))]
    srcs = [[i for i in range(len(sc.views)) if i != r] for r in range(3)]
    with DepthMapPool(max_active_jobs=4, use_graphs=use_graphs) as pool:
        add_scene(pool, sc, 0)
        jobs = [pool.submit(opts[0], 0, srcs[0])]
        pool.step()
        pool.step()
        jobs += [pool.submit(opts[r], r, srcs[r]) for r in (1, 2)]
        pool.run_until_done(jobs)
        maps = [pool.maps(j) for j in jobs]
    with _form(PIXEL):
        for r in range(3):
            assert_same(maps[r], engine_maps(opts[r], problem_from_scene(sc, ref=r)))


def test_launch_shapes_of_small_images_with_a_thread_per_pixel():
    """Every block shape, with and without tile descriptors, on an image that the
    size would send to the spread form. The tile of 64 pixels a row is 140 columns
    wide, wider than the image: it takes no descriptor."""
    scene = small_planes(seed=12, w=100, h=76, f=80.0)
    opt = photometric_options(scene, iters=5)
    problem = problem_from_scene(scene)
    want = engine_maps(opt, problem)
    with _form(PIXEL):
        for block_x in (8, 16, 32, 64):
            for tma in (True, False):
                with PatchMatchACMMCuda(opt, problem) as pm:
                    pm.SetTuning(block_x, tma, 1, False)
                    pm.Run()
                    assert pm.Tuning()["ref_tile_tma"] == (tma and block_x < 64)
                    np.testing.assert_array_equal(pm.GetDepthMap(), want["depth"])
                    np.testing.assert_array_equal(pm.GetCostMap(), want["cost"])
