"""The engine's frontier queues at their edges: objects of one and two voxels' width, frontiers that just fill a queue,
frontiers that spill past it in the floods and in the invalidation, and re-claimed voxels, each with every object
on one CTA and on clusters. A CTA queues 6144 pairs of a flood and 1754 of an invalidation, a cluster of four or eight as
many times more; a solid box flooded from a corner has a frontier of three times its face. Skeletons must be the
oracle's bit for bit."""
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
    if name == "box":  # a frontier of 6000 voxels: one CTA's queue
        return np.asfortranarray(np.pad(np.ones((44, 46, 45), np.uint16), 1))
    if name == "block":  # frontiers of 11000 voxels: past one CTA's queue
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


@pytest.mark.parametrize("copies,edge", [(1, 148), (17, 92)], ids=["cluster of 8", "clusters of 4"])
def test_frontiers_past_a_clusters_queues(gpu, monkeypatch, copies, edge):
    """Boxes whose frontiers (65 000 and 25 000 voxels) are past the queues of eight and of four CTAs, so that they spill to
    the object's lists; of seventeen objects none holds the sixteenth of the foreground that calls for eight."""
    monkeypatch.setenv("BROOK_B200_PREPARE_CLUSTER_VOXELS", "1")
    monkeypatch.setenv("BROOK_B200_TRACE_CLUSTER_VOXELS", "1")
    labels = np.asfortranarray(np.concatenate([np.pad(np.ones((edge,) * 3, np.uint8), 1)] * copies, axis=2))
    opts = dict(teasar_params=dict(PARAMS, const=60), anisotropy=(1, 1, 1), dust_threshold=0, fix_borders=False)
    expected = oracle.skeletonize(labels, threads=8, **opts)
    assert_same(bk().skeletonize(labels, output="packed", **opts), expected, f"{copies} of {edge}")


@pytest.mark.parametrize("cluster_voxels", ["1", "100000000"])
@pytest.mark.parametrize("spacing", [(1, 1, 40), (40, 1, 1)])
def test_reclaimed_voxels_past_their_list(gpu, monkeypatch, spacing, cluster_voxels):
    """A band re-claims up to a tenth of a porous object's voxels at these spacings, more than are listed: at its boundary
    every waiting voxel is looked at anew."""
    monkeypatch.setenv("BROOK_B200_PREPARE_CLUSTER_VOXELS", cluster_voxels)
    monkeypatch.setenv("BROOK_B200_TRACE_CLUSTER_VOXELS", cluster_voxels)
    labels = np.asfortranarray((np.random.default_rng(3).random((40, 40, 40)) < 0.4).astype(np.uint8))
    opts = dict(teasar_params=dict(PARAMS, const=300), anisotropy=spacing, dust_threshold=0)
    expected = oracle.skeletonize(labels, threads=8, **opts)
    assert_same(bk().skeletonize(labels, output="packed", **opts), expected, f"{spacing}")


def test_soma_seeds_past_a_queue(gpu, monkeypatch):
    """A soma's seeds (more voxels than a CTA queues) all enter its flood's first frontier, on one CTA."""
    from test_oracle_golden import SOMA_PARAMS, _soma_with_processes

    monkeypatch.setenv("BROOK_B200_PREPARE_CLUSTER_VOXELS", "100000000")
    monkeypatch.setenv("BROOK_B200_TRACE_CLUSTER_VOXELS", "100000000")
    labels = _soma_with_processes()
    opts = dict(teasar_params=SOMA_PARAMS, dust_threshold=0, fix_borders=False)
    assert_same(bk().skeletonize(labels, output="packed", **opts), oracle.skeletonize(labels, threads=8, **opts), "soma")
