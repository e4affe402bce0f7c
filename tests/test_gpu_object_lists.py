"""The objects' voxel lists of a batch whose volumes begin anywhere in a block of 4096 voxels (the unit by which a voxel's
volume is looked up), several of them in one block and one over many; and target orders among many equal distances, with
the sorted bits trimmed to the distances that the spacing allows and, for spacings 1e4 times apart, whole. Skeletons must
be the oracle's bit for bit."""
import numpy as np
import pytest

from oracle import oracle
from test_gpu_parity import assert_same, bk

pytestmark = pytest.mark.gpu

PARAMS = dict(scale=1.0, const=4, pdrf_scale=100000, pdrf_exponent=4)


def _blocks(shape, seed):
    """Solid boxes (equal distances everywhere) of several labels with background between them."""
    rng = np.random.default_rng(seed)
    v = np.zeros(shape, np.uint16, order="F")
    for label in range(1, 6):
        lo = [int(rng.integers(0, max(1, n - 2))) for n in shape]
        hi = [min(n, a + int(rng.integers(2, max(3, n)))) for a, n in zip(lo, shape)]
        v[tuple(slice(a, b) for a, b in zip(lo, hi))] = label
    return v


@pytest.mark.parametrize("aniso", [(1, 1, 1), (1, 2, 5), (0.001, 1, 20)])
def test_batch_lists_match_oracle(gpu, aniso):
    shapes = [(16, 16, 16), (15, 13, 21), (17, 241, 1), (16, 256, 1), (1, 7, 585), (40, 33, 29), (9, 9, 50)]
    volumes = [_blocks(s, i) for i, s in enumerate(shapes)]
    params = dict(PARAMS, const=4 * float(np.median(aniso)))
    got = bk().skeletonize_batch(volumes, output="packed", teasar_params=params, anisotropy=aniso, dust_threshold=3)
    assert len(got) == len(volumes)
    for i, volume in enumerate(volumes):
        expected = oracle.skeletonize(volume, teasar_params=params, anisotropy=aniso, dust_threshold=3)
        assert_same(got[i], expected, str(shapes[i]))


def test_background_only_tail(gpu):
    """An object in the first and the last voxels of a volume with whole blocks of background between."""
    v = np.zeros((64, 64, 9), np.uint32, order="F")
    v[:5, :4, 0] = 3
    v[-6:, -5:, -1] = 7
    opts = dict(teasar_params=PARAMS, anisotropy=(1, 1, 1), dust_threshold=3)
    assert_same(bk().skeletonize(v, output="packed", **opts), oracle.skeletonize(v, **opts), "two corners")
