"""Where an engine's device memory comes from: what callers on other devices, in
other processes and on other threads may do with its maps and while it closes."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from sensemap_b200 import _native as N
from sensemap_b200 import synthetic as syn
from sensemap_b200.cross_filter import CrossFilterCuda
from sensemap_b200.fusion import FusionOptions, StereoFusion
from sensemap_b200.init_maps import init_depth_from_sparse_points
from sensemap_b200.patch_match import PatchMatchACMMCuda, PatchMatchOptions, Problem, View
from sensemap_b200.pool import DepthMapPool
from tests.helpers import (filter_api_inputs, filter_set, photometric_options, problem_from_scene,
                           small_planes)

pytestmark = pytest.mark.gpu

MAPS = ("depth", "normal", "conf", "cost", "view_sel")


def _engine(iters=1, **size):
    scene = small_planes(seed=11, **size)
    pm = PatchMatchACMMCuda(photometric_options(scene, iters=iters), problem_from_scene(scene))
    pm.Run()
    pm.Synchronize()
    return pm


def test_device_maps_can_be_exported_to_another_process():
    driver = C.CDLL("libcuda.so.1")
    with _engine() as pm:
        maps = pm.DeviceMaps()
        for name in MAPS:
            address = C.cast(getattr(maps, name), C.c_void_p).value
            handle = (C.c_char * 64)()
            assert driver.cuIpcGetMemHandle(handle, C.c_uint64(address)) == 0, name
            base, size = C.c_uint64(), C.c_size_t()
            assert driver.cuMemGetAddressRange_v2(C.byref(base), C.byref(size), C.c_uint64(address)) == 0
            assert base.value == address, name  # a handle opens at the map itself


def test_given_maps_are_not_left_to_the_next_engine():
    """Blocks of closed engines serve later ones, but not those whose address a
    caller was given: it may still be read elsewhere until the close has returned."""
    lib = N.lib()
    N.check(lib.smvs_cross_filter_release_cache(-1))
    with _engine(w=320, h=240) as a:
        first = a.GetDepthMap()
        given = a.DeviceMaps()
        other = _engine(w=320, h=240)  # takes blocks of its own
        assert C.cast(other.DeviceMaps().depth, C.c_void_p).value != C.cast(given.depth, C.c_void_p).value
        other.close()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        with _engine(w=320, h=240) as pm:
            assert (pm.GetDepthMap() == first).all()
    N.check(lib.smvs_cross_filter_release_cache(-1))
    assert torch.cuda.mem_get_info()[0] >= before


def test_blocks_left_to_the_next_engine_are_bounded():
    """The blocks of ten engines of different sizes together hold more than their
    bound of 1 GiB; what is above it goes back to the device."""
    lib = N.lib()
    N.check(lib.smvs_cross_filter_release_cache(-1))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    scene = small_planes(seed=11, w=32, h=24, n_src=8)
    for k in range(10):
        w, h = 1600 + 160 * k, 1200 + 120 * k
        views = [View(np.zeros((h, w), np.uint8), v.K, v.R, v.T) for v in scene.views]
        problem = Problem(0, list(range(1, 9)), views)
        PatchMatchACMMCuda(photometric_options(scene, iters=0), problem).close()
    assert before - torch.cuda.mem_get_info()[0] <= (4 << 30) + (256 << 20)
    N.check(lib.smvs_cross_filter_release_cache(-1))
    assert before - torch.cuda.mem_get_info()[0] <= 256 << 20


def test_closing_an_engine_leaves_another_threads_capture_alone():
    x = torch.zeros(256, device="cuda")
    engines = [_engine() for _ in range(2)]
    engines[1].DeviceMaps()  # its maps are freed, not kept
    torch.cuda.synchronize()
    graph, failed = torch.cuda.CUDAGraph(), []

    def close_all():
        try:
            for pm in engines:
                pm.close()
            _engine().close()
        except Exception as error:  # noqa: BLE001
            failed.append(error)

    with torch.cuda.stream(torch.cuda.Stream()):
        graph.capture_begin(capture_error_mode="thread_local")
        x.add_(1)
        thread = threading.Thread(target=close_all)
        thread.start()
        thread.join()
        x.add_(1)
        graph.capture_end()
    assert not failed
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 2).all()


def _fusion():
    scene = syn.planes_scene(seed=3, width=90, height=70, focal=72.0, num_src=3)
    images, overlaps = syn.fusion_inputs(scene, seed=1)
    with StereoFusion(FusionOptions(), images, overlaps) as f:
        f.Run()
        assert f.RemoveOutliers() >= 0


def _cross_filter():
    _, views, problems = filter_set(n_views=3, w=64, h=48)
    cf = CrossFilterCuda(PatchMatchOptions(), *filter_api_inputs(views, problems))
    cf.Run()
    cf.close()


def _initial_map():
    scene = small_planes(seed=11, w=64, h=48)
    v = scene.views[0]
    init_depth_from_sparse_points(64, 48, v.K, v.R, v.T, np.random.default_rng(0).random((50, 3)))


def _pool():
    scene = small_planes(seed=11, w=64, h=48)
    with DepthMapPool(max_active_jobs=2) as pool:
        for i, v in enumerate(scene.views):
            pool.add_view(i, View(v.image, v.K, v.R, v.T))
        job = pool.submit(photometric_options(scene, iters=1), 0, [1, 2, 3, 4])
        pool.run_until_done([job])
        pool.keep_maps(job)


def _next_engine():
    _engine(w=64, h=48).close()


@pytest.mark.parametrize("call", [_fusion, _cross_filter, _initial_map, _pool, _next_engine])
def test_a_full_device_takes_back_what_closed_engines_left(call):
    """An engine of 1600x1200 leaves over 64 MiB to the next one; on a device that
    is full as long as it does, every kind of call gets its memory all the same."""
    lib = N.lib()
    scene = small_planes(w=32, h=24)
    views = [View(np.zeros((1200, 1600), np.uint8), v.K, v.R, v.T) for v in scene.views]
    PatchMatchACMMCuda(photometric_options(scene, iters=0), Problem(0, [1, 2, 3, 4], views)).close()
    N.check(lib.smvs_test_device_full(64 << 20))
    try:
        call()
    finally:
        N.check(lib.smvs_test_device_full(0))
