"""Renders of different tile counts from several host threads at once: the
histogram's shared memory, sized by the tile count, is one limit of the kernel
for all of them."""
import threading

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import gpu_helpers as gh  # noqa: E402
from word2world_b200 import _C, camera, scenes  # noqa: E402

# 9600, 16384, 8300 and 25600 tiles: 1024 threads to a histogram block, 45 to 110 KB of counters
SIZES = [(2048, 1200), (2048, 2048), (1328, 1600), (2560, 2560)]


def _args(W, H):
    m, o, s, q, sh = (gh.dev(a) for a in scenes.make_scene(500, seed=W + H, layout="ball",
                                                            log_scale=(-5.0, -3.0)).activate())
    cam = camera.orbit_camera(33.0, 5.0, 2.5, W, H)
    v, p, c = (gh.dev(a) for a in (cam.viewmatrix, cam.projmatrix, cam.campos))
    return lambda: _C.rasterize_gaussians(sh, float(cam.focal_y), s, m, p, 3, o, q, c, v, float(cam.focal_x), H, W,
                                          None, True)


def test_threads_with_their_own_tile_counts():
    calls = [_args(*size) for size in SIZES]
    want = [call()[:4] for call in calls]
    torch.cuda.synchronize()
    wrong, start = [], threading.Barrier(len(calls))

    def work(i):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                start.wait()
                got = [calls[i]()[:4] for _ in range(12)]
                stream.synchronize()
            for R, *images in got:
                if R != want[i][0] or not all(torch.equal(a, b) for a, b in zip(images, want[i][1:])):
                    wrong.append(SIZES[i])
        except Exception as e:  # a refused launch
            wrong.append((SIZES[i], repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
    _C.check_device_errors()
