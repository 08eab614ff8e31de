"""The voxel field's two routes (a fixed number of block slots per Gaussian, and
pairs counted first) and its two voxels per thread, at the sizes where they
change, against the numpy restatement."""
import os
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
from oracle import voxel as ovox  # noqa: E402
from word2world_b200 import voxel  # noqa: E402

pytestmark = pytest.mark.gpu


def _gaussians(n, seed):
    rng = np.random.default_rng(seed)
    means = rng.uniform(-1.0, 1.0, size=(n, 3)).astype(np.float32)
    means[: n // 8] = np.round(means[: n // 8] * 4) / 4  # on block bounds
    a = rng.normal(size=(n, 3, 3)) * 0.08
    s = a @ a.transpose(0, 2, 1) + 1e-3 * np.eye(3)
    covs = np.stack([s[:, 0, 0], s[:, 0, 1], s[:, 0, 2], s[:, 1, 1], s[:, 1, 2], s[:, 2, 2]], 1).astype(np.float32)
    return means, covs, rng.uniform(0.0, 1.0, size=(n, 1)).astype(np.float32)


def _field(means, covs, opac, r, b, relax):
    t = lambda x: torch.from_numpy(x).cuda()
    return voxel.voxel_field(t(means), t(covs), t(opac), r, b, relax).cpu().numpy()


def _close(got, want, n):
    # a sum of up to n positive terms in 32 bits, each a few roundings from its own value
    np.testing.assert_allclose(got, want, rtol=2e-5 + n * 2.0 ** -24, atol=1e-6)


@pytest.mark.parametrize("n,r,b,relax", [
    (1, 2, 1, 0.0),      # one pair of voxels per axis, the second in the block past the last
    (257, 9, 3, 0.0),    # an odd grid: the last layer has no second voxel; a ragged block of threads
    (500, 17, 5, 0.5),   # grown bounds that meet: three blocks an axis
    (300, 15, 7, 1.0),   # voxel pairs that straddle blocks
    (2048, 8, 7, 3.0),   # 2^20 slots: the last size with slots
    (2049, 8, 7, 3.0),   # one more Gaussian: counted
])
def test_routes_match(n, r, b, relax):
    means, covs, opac = _gaussians(n, seed=n + r)
    _close(_field(means, covs, opac, r, b, relax), ovox.voxel_field(means, covs, opac, r, b, relax), n)


def test_mean_without_a_number_leaves_the_rest():
    # it takes more blocks than it has slots (0 to 2 of each axis), and is counted instead
    n, r, b = 64, 16, 8
    means, covs, opac = _gaussians(n, seed=3)
    means[5] = np.nan
    got = _field(means, covs, opac, r, b, 0.1)
    keep = np.arange(n) != 5
    want = ovox.voxel_field(means[keep], covs[keep], opac[keep], r, b, 0.1)
    _close(got[6:, 6:, 6:], want[6:, 6:, 6:], n)
