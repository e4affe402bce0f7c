"""The railroad's bands when one is empty. A band past the deferred voxels is named by the least offer made beyond the
band before it; the voxel that got that offer may have been improved into that band since, and then the named band can
hold nothing while deferred voxels wait behind it. A model of the bands shows that the volumes here have such bands and
that a thread which takes the next band's end for the empty band's own loses the waiting voxels and with them the path;
the skeletons traced on one CTA and on clusters of four and eight must be the oracle's bit for bit."""
import numpy as np
import pytest

from oracle import oracle

PARAMS = dict(scale=1.5, const=100, pdrf_scale=100000, pdrf_exponent=4)
OPTS = dict(teasar_params=PARAMS, anisotropy=(4, 4, 40), dust_threshold=0)
RAIL_BAND = np.float32(0.5)  # engine.hpp: kRailBand


def _porous(seed):
    return np.asfortranarray((np.random.default_rng(seed).random((28, 28, 28)) < 0.62).astype(np.uint8))


def _neighbours(ids):
    """The object voxels' places in the flat volume and, per voxel, its 26 neighbours' indices of the same id or -1."""
    flat = np.flatnonzero(ids.ravel(order="F"))
    index = np.full(ids.size, -1)
    index[flat] = np.arange(len(flat))
    own = ids.ravel(order="F")[flat]
    at = np.stack(np.unravel_index(flat, ids.shape, order="F"), 1)
    columns = []
    for step in np.ndindex(3, 3, 3):
        if step == (1, 1, 1):
            continue
        q = at + np.array(step) - 1
        inside = ((q >= 0) & (q < ids.shape)).all(1)
        g = np.where(inside, q[:, 0] + ids.shape[0] * (q[:, 1] + ids.shape[1] * q[:, 2]), 0)
        columns.append(np.where(inside & (ids.ravel(order="F")[g] == own), index[g], -1))
    return index, np.stack(columns, 1)


def _railroad(neighbours, penalty, target, late=False):
    """The nearest rail's distance (None: no rail found) and the empty bands with voxels waiting behind them, by
    synchronous rounds. `late`: an empty band's end is read after it has been overwritten with the next one's."""
    inf, none = np.float32(np.inf), np.zeros(0, np.int64)
    dist = np.full(len(penalty), inf, np.float32)
    dist[target] = 0
    if penalty[target] == 0:
        return np.float32(0), 0
    end, nearest, empty = max(RAIL_BAND * penalty[target], np.float32(1e-30)), inf, 0
    front, far, least = np.array([target]), none, (inf, np.float32(0))  # least: the nearest deferred offer, its penalty
    while True:
        rounds = 0
        while len(front):
            rounds += 1
            ok = neighbours[front] >= 0
            v, x = neighbours[front][ok], np.repeat(dist[front][:, None], 26, 1)[ok]
            f = penalty[v]
            c = x + f
            c = np.where((c == x) & (f > 0), np.nextafter(x, inf), c)
            want = (c < dist[v]) & (c <= nearest)
            v, f, c = v[want], f[want], c[want]
            fresh, rail = np.isinf(dist[v]), f == 0
            nearest = min([nearest, *c[rail]])
            beyond = (c > end) & ~rail
            least = min([least, *zip(c[beyond], f[beyond])])
            np.minimum.at(dist, v, c)
            far, front = np.union1d(far, v[beyond & fresh]), np.unique(v[~beyond & ~rail])
        if nearest < inf and (nearest <= end or least[0] > nearest):
            return nearest, empty
        if least[0] == inf:
            return None, empty
        following = least[0] + max(RAIL_BAND * least[1], np.float32(5e-4) * least[0])
        empty += rounds == 0 and bool((dist[far] > end).any())
        if late and rounds == 0:
            end = following
        far = far[dist[far] > end]
        front, far = far[dist[far] <= following], far[dist[far] > following]
        least = min([(inf, np.float32(0)), *zip(dist[far], penalty[far])])
        end = following


@pytest.mark.parametrize("seed", [7, 13])
def test_empty_bands_hide_waiting_voxels(seed):
    run = oracle.skeletonize(_porous(seed), threads=8, stages=True, **OPTS)
    index, neighbours = _neighbours(run.field("cc"))
    penalty = run.field("pdrf").ravel(order="F")[index >= 0]
    roots = run.array("roots")
    penalty[index[roots[roots >= 0]]] = 0
    paths = np.split(run.array("paths"), run.array("path_offsets")[1:-1])
    empty = lost = 0
    for path in paths:
        target = index[path[0]]
        found, bands = _railroad(neighbours, penalty, target)
        assert found is not None
        empty += bands
        lost += bands > 0 and _railroad(neighbours, penalty, target, late=True)[0] != found
        penalty[index[path]] = 0
    assert empty > 0 and lost > 0


@pytest.mark.gpu
@pytest.mark.parametrize("copies,cluster_voxels", [(1, "100000000"), (1, "1"), (17, "1")],
                         ids=["lone", "cluster of 8", "clusters of 4"])
@pytest.mark.parametrize("seed", [7, 13])
def test_empty_bands_match_oracle(gpu, monkeypatch, seed, copies, cluster_voxels):
    from test_gpu_parity import assert_same, bk

    monkeypatch.setenv("BROOK_B200_PREPARE_CLUSTER_VOXELS", cluster_voxels)
    monkeypatch.setenv("BROOK_B200_TRACE_CLUSTER_VOXELS", cluster_voxels)
    # 17 objects of one size: none holds the sixteenth of the foreground that calls for the wide clusters
    labels = np.asfortranarray(np.concatenate([np.pad(_porous(seed), ((0, 0), (0, 0), (0, 1)))] * copies, axis=2))
    expected = oracle.skeletonize(labels, threads=8, **OPTS)
    for _ in range(3):
        assert_same(bk().skeletonize(labels, output="packed", **OPTS), expected, f"{seed} x {copies}")
