"""Where an engine's device memory comes from: what callers on other devices, in
other processes and on other threads may do with its maps and while it closes."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from sensemap_b200 import _native as N
from sensemap_b200.patch_match import PatchMatchACMMCuda, Problem, View
from tests.helpers import photometric_options, problem_from_scene, small_planes

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
