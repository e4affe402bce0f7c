"""Calls with many tiny objects, which run on CTAs of 256 threads after the others': objects of one voxel to the 4095 that
still count as tiny (frontiers past the small queues among them), beside larger ones; calls just below and at the 1024
tiny objects that call for it, and with a larger object that holds more than they do. Skeletons must be the oracle's bit for bit."""
import numpy as np
import pytest

from oracle import oracle
from test_gpu_parity import assert_same, bk

pytestmark = pytest.mark.gpu

PARAMS = dict(scale=1.5, const=8, pdrf_scale=100000, pdrf_exponent=4)


def _cells(count, pitch=18, across=11):
    """`count` objects in cells of a grid, of kinds by turns: boxes of 15 x 16 x 17 (4080 voxels), plates, lines, porous
    blocks, single voxels; and two large objects over the planes beyond the grid."""
    rng = np.random.default_rng(count)
    v = np.zeros((across * pitch, across * pitch, across * pitch + 24), np.uint16, order="F")
    for i in range(count):
        x, y, z = (pitch * int(k) for k in np.unravel_index(i, (across,) * 3))
        cell = v[x:x + pitch - 1, y:y + pitch - 1, z:z + pitch - 1]
        kind = i % 5
        if kind == 0:
            cell[:15, :16, :17] = i + 1
        elif kind == 1:
            cell[:, 3, :] = i + 1
        elif kind == 2:
            cell[5, 5, :] = i + 1
        elif kind == 3:
            cell[rng.random(cell.shape) < 0.6] = i + 1
        else:
            cell[0, 0, 0] = i + 1
    v[2:-2, 2:60, -20:-2] = 60000
    v[2:-2, 70:-2, -20:-2] = 60001
    return v


@pytest.mark.parametrize("count,fix_branching,aniso", [(1331, True, (1, 1, 1)), (1331, False, (1, 1, 1)),
                                                       (1331, True, (4, 4, 40))])
def test_many_tiny_objects_match_oracle(gpu, count, fix_branching, aniso):
    labels = _cells(count)
    opts = dict(teasar_params=dict(PARAMS, const=8 * aniso[1]), anisotropy=aniso, dust_threshold=0,
                fix_branching=fix_branching)
    expected = oracle.skeletonize(labels, threads=8, **opts)
    for graph in ("1", "0"):
        with pytest.MonkeyPatch.context() as m:
            m.setenv("BROOK_B200_GRAPH", graph)
            assert_same(bk().skeletonize(labels, output="packed", **opts), expected, f"{count}, graph {graph}")


@pytest.mark.parametrize("count", [1023, 1024, 1030])
def test_about_as_many_tiny_objects_as_call_for_small_ctas(gpu, count):
    labels = np.zeros((10 * 12, 10 * 11, 10 * 10), np.uint16, order="F")
    for i in range(count):
        x, y, z = (int(k) for k in np.unravel_index(i, (12, 11, 10)))
        labels[10 * x:10 * x + 2 + i % 7, 10 * y:10 * y + 1 + i % 5, 10 * z:10 * z + 2 + i % 8] = i + 1
    opts = dict(teasar_params=PARAMS, anisotropy=(1, 1, 1), dust_threshold=0)
    for low in (0, 30):  # only tiny objects; too few once the dust is gone
        opts["dust_threshold"] = low
        assert_same(bk().skeletonize(labels, output="packed", **opts), oracle.skeletonize(labels, threads=8, **opts),
                    f"{count}, dust {low}")
    opts["dust_threshold"] = 0
    slab = np.asfortranarray(np.pad(labels, ((0, 0), (0, 0), (0, 20))))
    slab[:, :, -18:] = 60000
    assert_same(bk().skeletonize(slab, output="packed", **opts), oracle.skeletonize(slab, threads=8, **opts), "slab")


def test_batch_of_tiny_and_large_objects(gpu):
    """Objects of a batch's volumes side by side in one schedule."""
    volumes = [_cells(700), _cells(600)[:, :, :120], np.asfortranarray(np.pad(np.ones((40, 30, 20), np.uint16), 1))]
    opts = dict(teasar_params=PARAMS, anisotropy=(1, 1, 1), dust_threshold=0)
    got = bk().skeletonize_batch(volumes, output="packed", **opts)
    for i, v in enumerate(volumes):
        assert_same(got[i], oracle.skeletonize(v, threads=8, **opts), str(i))
