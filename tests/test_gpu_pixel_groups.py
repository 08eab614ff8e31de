"""The per-pixel and per-Gaussian kernels and the sort where their paths change:
group sizes of the lane-per-entry evaluation, the mask window, state aligned to
16 bytes only, SH rows that cannot be copied in 16-byte pieces, tile sizes of
small sorts, many tiles in the histogram."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import gpu_helpers as gh  # noqa: E402
import parity  # noqa: E402
from test_gpu_parity import _check_forward, _grads, _orc, _setup  # noqa: E402
from word2world_b200 import _C, camera, scenes  # noqa: E402


def _layers(P, W=21, H=19):
    """P faint Gaussians that all reach every block of a small ragged image."""
    (m, o, s, q, sh), cam = _setup(P=P, seed=P, W=W, H=H, log_scale=(-1.2, -0.8), layout="ball")
    return (m * 0.3, np.full_like(o, 0.03), s, q, sh), cam


# one entry; the edges of 8, 16 and 32 lanes; more than one group; the 512-position window and its edge
@pytest.mark.parametrize("P", [1, 8, 9, 16, 17, 32, 33, 512, 513, 545])
def test_group_sizes(P):
    arrays, cam = _layers(P)
    _check_forward(gh.forward(arrays, cam), _orc(arrays, cam))
    for mode in ("reference", "exact"):
        mine, orc = _grads(arrays, cam, mode)
        for k in parity.GRAD_NAMES:
            c = parity.grad_check(mine[k], orc[k], abs_sum=orc.get("abs_" + k))
            assert c["norm_rel"] <= 1e-4, (P, mode, k, c)
            if mode == "reference":
                assert c["n_bad"] == 0, (P, mode, k, c)


def _shift16(t):
    buf = torch.empty(t.numel() + 512, dtype=torch.uint8, device="cuda")
    out = buf[16:16 + t.numel()]
    assert out.data_ptr() % 32 == 16
    return out.copy_(t)


def test_state_aligned_to_16_bytes():
    arrays, cam = _setup(P=3000, seed=4, size=160)
    f = gh.forward(arrays, cam)
    W, H = cam.width, cam.height
    rng = torch.from_numpy(f["ranges"].view(np.int32)).cuda()
    pl = torch.from_numpy(f["point_list"].view(np.int32)).cuda()
    a = _C.blend(f["_tensors"]["geom"], 3000, rng, pl, H, W, None)
    b = _C.blend(_shift16(f["_tensors"]["geom"]), 3000, rng, pl, H, W, None)
    for x, y in zip(a[:3], b[:3]):
        assert torch.equal(x, y)
    g = np.random.default_rng(0).normal(size=(3, H, W)).astype(np.float32)
    for mode in (0, 1):
        want = gh.backward(f, arrays, cam, g, grad_mode=mode)
        shifted = dict(f, _tensors=dict(f["_tensors"], geom=_shift16(f["_tensors"]["geom"])))
        got = gh.backward(shifted, arrays, cam, g, grad_mode=mode)
        for k in parity.GRAD_NAMES:
            c = parity.grad_check(got[k], want[k], row_rtol=parity.SAME_IMPL_ROW_RTOL)
            assert c["norm_rel"] <= 1e-5 and c["n_bad"] == 0, (mode, k, c)


# a full warp, a partial one beside it, and every lane's row at its own address
@pytest.mark.parametrize("P", [31, 32, 97])
def test_raw_rows_off_16_bytes(P):
    sc = scenes.make_scene(P, seed=P, layout="ball", log_scale=(-2.5, -1.5))
    m, o, s, q, sh = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in sc.activate())
    W = H = 64
    cam = camera.orbit_camera(20.0, 5.0, 2.5, W, H)
    v, pr, cp = (gh.dev(x) for x in (cam.viewmatrix, cam.projmatrix, cam.campos))
    logit, svec = torch.logit(o.clamp(1e-3, 1 - 1e-3)).contiguous(), s.log().contiguous()
    dc, ac = sh[:, :1].contiguous(), sh[:, 1:].contiguous()
    bg, e = torch.ones(3, device="cuda"), torch.empty(0, device="cuda")
    up = torch.from_numpy(np.random.default_rng(1).normal(size=(3, H, W)).astype(np.float32)).cuda()

    def off(t):  # the same values four bytes further
        return torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view(t.shape)

    outs = []
    for f in (lambda t: t, off):
        x = [f(t) for t in (m, dc, ac, logit, svec, q.contiguous())]
        R, col, dep, al, rad, geom, binb, img = _C.rasterize_gaussians_raw(*x, v, pr, cp, cam.focal_x, 3, H, W, bg, True)
        g = _C.rasterize_gaussians_backward_raw(bg, *x, rad, v, pr, cp, cam.tanfovx, cam.tanfovy, 3, up, e, e, geom, R,
                                                binb, img, al)
        outs.append((col, dep, al, rad, g))
    for a, b in zip(outs[0][:4], outs[1][:4]):
        assert torch.equal(a, b)
    for a, b in zip(outs[0][4], outs[1][4]):
        if a is None or a.numel() == 0:
            continue
        c = parity.grad_check(b.reshape(P, -1).cpu().numpy(), a.reshape(P, -1).cpu().numpy(),
                              row_rtol=parity.SAME_IMPL_ROW_RTOL)
        assert c["norm_rel"] <= 1e-5 and c["n_bad"] == 0, c


# tiles of 2048 keys, their remainders, the last size that has them and the first that has not
@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 700000, 700001])
@pytest.mark.parametrize("bits", [5, 27, 44])
def test_small_sorts(n, bits):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64) & np.uint64(~0xf0 & ((1 << bits) - 1))
    vals = np.arange(n, dtype=np.int32)
    k, v = _C.sort_pairs_u64(torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(vals).cuda(), 0, bits)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k.cpu().numpy().view(np.uint64), keys[order])
    assert np.array_equal(v.cpu().numpy(), vals[order])


# tile counts beside the digits in shared memory, alone in most of it, and past it (16 by 16 pixels a tile)
@pytest.mark.parametrize("W,H", [(1024, 2048), (1024, 2064), (3500, 3600), (3600, 3600)])
def test_tile_counts(W, H):
    arrays = scenes.make_scene(700, seed=9, layout="ball", log_scale=(-5.0, -2.0)).activate()
    cam = camera.orbit_camera(33.0, 5.0, 2.5, W, H)
    f = gh.forward(arrays, cam, degree=0)
    tiles = (f["keys"] >> np.uint64(32)).astype(np.int64)
    T = ((W + 15) // 16) * ((H + 15) // 16)
    assert np.all(np.diff(f["keys"].view(np.int64)) >= 0)
    first, count = np.searchsorted(tiles, np.arange(T)), np.bincount(tiles, minlength=T)
    want = np.where(count[:, None] > 0, np.stack([first, first + count], 1), 0).astype(np.uint32)
    assert np.array_equal(f["ranges"], want)
