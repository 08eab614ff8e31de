"""A batch whose list is emitted in depth order, and tile counts that fill most of
a histogram block's shared memory."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import gpu_helpers as gh  # noqa: E402
from test_gpu_pixel_groups import test_tile_counts as check_tile_counts  # noqa: E402
from word2world_b200 import _C, camera, scenes  # noqa: E402
from word2world_b200.batch import BatchRenderer, Scene, View  # noqa: E402


def test_batch_in_depth_order():
    """Its list is the views' own lists, of fewer than the rule's 2M instances each (sorted by the full key), in turn."""
    specs = [(6007, 640, 640, 2.5), (9001, 500, 700, 2.4), (4001, 801, 603, 2.5)]
    arrays = [scenes.make_scene(P, seed=21, layout="ball", log_scale=(-3.5, -2.0)).activate() for P, *_ in specs]
    cams = [camera.orbit_camera(33.0, 5.0, r, W, H) for _, W, H, r in specs]
    res = BatchRenderer().forward([Scene.from_arrays(a, "cuda") for a in arrays],
                                  [View(i, c, (1.0, 1.0, 1.0)) for i, c in enumerate(cams)])
    _C.check_device_errors()
    R = res.state["R"]
    P = [spec[0] for spec in specs]
    assert R >= 2_000_000 and R >= 8 * sum(P)
    ids, nc = [], []
    for v, (a, c) in enumerate(zip(arrays, cams)):
        f = gh.forward(a, c)
        assert f["num_rendered"] < 2_000_000
        ids.append(f["point_list"].astype(np.int64) + sum(P[:v]))
        nc.append(f["n_contrib"].reshape(-1))
        for mine, want in ((res.color[v], f["color"]), (res.depth[v], f["depth_img"]), (res.alpha[v], f["alpha"])):
            assert np.array_equal(mine.cpu().numpy().reshape(want.shape), want), v
    off = _C.binning_offset(R, 16, 16, "vals_a")  # does not depend on the tiles
    got = res.state["binb"][off:off + 4 * R].cpu().numpy().view(np.uint32)
    assert np.array_equal(got, np.concatenate(ids))
    nc = np.concatenate(nc)
    assert np.array_equal(res.state["img"][:4 * len(nc)].cpu().numpy().view(np.uint32), nc)


# 1024 threads to a histogram block: one round of its closing block, the first size of two, all the shared memory
@pytest.mark.parametrize("W,H,tiles", [(2048, 2048, 16384), (2048, 2064, 16512), (3488, 3600, 49050), (4096, 3072, 49152)])
def test_many_tiles(W, H, tiles):
    assert ((W + 15) // 16) * ((H + 15) // 16) == tiles
    check_tile_counts(W, H)
