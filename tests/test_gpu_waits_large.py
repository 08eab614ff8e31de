"""The bounded waits that only large calls have, made to run out as in
test_gpu_waits.py: the depth-ordered emission's sort of its Gaussians and its
scan, and the sorts' large tiles (5120 64-bit keys, 6144 32-bit keys)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import gpu_helpers as gh  # noqa: E402
from test_gpu_waits import STAGE_SORT, hooked  # noqa: E402
from word2world_b200 import _C, camera, scenes  # noqa: E402

STAGE_EMIT_SORT, STAGE_EMIT = 3, 4


def test_large_sort_tiles():
    n = 700001 + 12 * 5120
    keys = np.random.default_rng(2).integers(0, 1 << 40, size=n).astype(np.uint64)
    k = torch.from_numpy(keys.view(np.int64)).cuda()
    v = torch.arange(n, dtype=torch.int32, device="cuda")
    with hooked(STAGE_SORT, 2):
        with pytest.raises(RuntimeError, match="timed out"):
            _C.sort_pairs_u64(k, v, 0, 40)
    ko, vo = _C.sort_pairs_u64(k, v, 0, 40)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(ko.cpu().numpy().view(np.uint64), keys[order])
    assert np.array_equal(vo.cpu().numpy(), order.astype(np.int32))


# 3001 Gaussians of 2.2M or more instances: two tiles of the depth sort, twelve blocks of the emission
@pytest.mark.parametrize("planned", [0, 1])
@pytest.mark.parametrize("stage,tile", [(STAGE_EMIT_SORT, 0), (STAGE_EMIT, 0), (STAGE_EMIT, 5), (STAGE_SORT, 0),
                                        (STAGE_SORT, 7)])
def test_depth_ordered_render(stage, tile, planned):
    arrays = scenes.make_scene(3001, seed=21, layout="ball", log_scale=(-3.0, -1.5)).activate()
    cam = camera.orbit_camera(33.0, 5.0, 2.5, 1024, 1030)
    with gh.tuned(planned_forward=planned):
        gh.forward(arrays, cam, degree=0)  # a planned render needs one of its size before it
        clean = gh.forward(arrays, cam, degree=0)
        assert clean["num_rendered"] >= 2_000_000
        with hooked(stage, tile):
            gh.forward(arrays, cam, degree=0)  # returns; its list is invalid
            with pytest.raises(RuntimeError, match="timed out"):
                _C.check_device_errors()
        again = gh.forward(arrays, cam, degree=0)
        _C.check_device_errors()
    for key in ("keys", "point_list", "ranges", "n_contrib", "color", "alpha"):
        assert np.array_equal(again[key], clean[key]), key
