"""The fusion paths that only large inputs take, against the oracle: closures
without the projection table (it would not fit), the replay without predecessor
lists (they would not fit or a seed has too many), clusters of more than 64
pixels and images whose seed grid is narrower than the predecessor window."""
import numpy as np
import pytest

import oracle.oracle as O
from sensemap_b200 import _native as N
from sensemap_b200 import synthetic as syn
from sensemap_b200.fusion import FusionOptions
from tests.test_fusion_gpu import _run, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,views,in_place,walk,options", [
    ((160, 120), 5, 1, 0, {}), ((160, 120), 5, 0, 1, {}), ((97, 61), 4, 1, 1, {"min_num_visible_images": 2}),
    ((36, 90), 4, 0, 0, {"min_num_visible_images": 1, "min_num_pixels": 2}),
    ((320, 240), 11, 0, 1, {}), ((240, 180), 9, 0, 0, {"max_reproj_error": 4.0, "max_traversal_depth": 400})])
def test_large_input_paths_match_oracle(size, views, in_place, walk, options):
    scene = syn.heightfield_scene(seed=9, width=size[0], height=size[1], focal=0.75 * size[0], num_src=views - 1,
                                  device="cuda")
    images, overlaps = syn.fusion_inputs(scene, seed=3)
    opts = FusionOptions(**options)
    N.check(N.lib().smvs_test_fusion_paths(in_place, walk))
    try:
        got = _run(opts, images, overlaps)
    finally:
        N.check(N.lib().smvs_test_fusion_paths(0, 0))
    want = O.fusion_run(opts, images, overlaps)
    assert len(want["points"]) > 20
    _same(got, want)
