"""The engine's frontier queues at their edges: objects of one and two voxels' width, frontiers that just fill a queue,
frontiers that spill past it in the floods and in the invalidation, and re-claimed voxels, each with every object
on one CTA and on a cluster. Skeletons must be the oracle's bit for bit."""
import numpy as np
import pytest

from oracle import oracle
from test_gpu_parity import assert_same, bk

pytestmark = pytest.mark.gpu

PARAMS = dict(scale=1.5, const=10, pdrf_scale=100000, pdrf_exponent=4)


def _volume(name):
    if name == "thin":  # a line, a plane and an isolated pair
        v = np.zeros((40, 36, 30), np.uint8)
        v[2:38, 3, 3] = 1
        v[2:38, 8:30, 10] = 2
        v[5, 5, 20:22] = 3
        return np.asfortranarray(v)
    if name == "box":  # frontiers of a few hundred voxels: a queue's size
        return np.asfortranarray(np.pad(np.ones((29, 27, 31), np.uint16), 1))
    if name == "block":  # frontiers of thousands: past every queue
        v = np.pad(np.ones((93, 61, 70), np.uint32), 1)
        v[40, 10:50, :] = 0  # a wall with a gap: claims that improve later
        return np.asfortranarray(v)
    rng = np.random.default_rng(11)  # porous: many sources, many re-claims
    v = (rng.random((57, 49, 44)) < 0.62).astype(np.uint8)
    return np.asfortranarray(v)


@pytest.mark.parametrize("cluster_voxels", ["1", "100000000"])
@pytest.mark.parametrize("aniso", [(1, 1, 1), (4, 4, 40)])
@pytest.mark.parametrize("name", ["thin", "box", "block", "porous"])
def test_queue_edges_match_oracle(gpu, monkeypatch, name, aniso, cluster_voxels):
    monkeypatch.setenv("BROOK_B200_PREPARE_CLUSTER_VOXELS", cluster_voxels)
    monkeypatch.setenv("BROOK_B200_TRACE_CLUSTER_VOXELS", cluster_voxels)
    labels = _volume(name)
    opts = dict(teasar_params=dict(PARAMS, const=10 if aniso[2] == 1 else 100), anisotropy=aniso, dust_threshold=0)
    expected = oracle.skeletonize(labels, threads=8, **opts)
    assert_same(bk().skeletonize(labels, output="packed", **opts), expected, name)
