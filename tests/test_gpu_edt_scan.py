"""The distance field's scans over whole lines against the oracle's envelope, bit for bit: lines at the edges of
a block of 32 voxels and of the near steps, solid runs without a wall, columns that do not fill a tile, spacings on
both sides of the rule that admits the scans, and a line too long for them."""
import ctypes

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _edt(labels, aniso, black_border):
    from brook_b200 import _native as n

    arr = ctypes.c_void_p()
    vol = n.host_volume(labels)
    n.check(n.load().brook_edt(n.context(0), ctypes.byref(vol), (ctypes.c_float * 3)(*aniso), int(black_border),
                               ctypes.byref(arr)))
    out = np.zeros(labels.shape, np.float32, order="F")
    n.check(n.lib.brook_array_copy_to_host(arr, out.ctypes.data, out.nbytes))
    n.lib.brook_array_destroy(arr)
    return out


def _labels(shape, kind):
    rng = np.random.default_rng(sum(shape))
    if kind == "solid":
        return np.ones(shape, np.uint32, order="F")
    if kind == "hole":  # one background voxel: nearly every voxel scans by blocks
        v = np.ones(shape, np.uint32, order="F")
        v[shape[0] // 2, shape[1] // 3, shape[2] - 1] = 0
        return v
    if kind == "noise":
        return np.asfortranarray(rng.integers(0, 3, shape).astype(np.uint32))
    # slabs of several labels, some over the volume's ends, with a few holes
    v = (np.add.outer(np.add.outer(np.arange(shape[0]) // 19, np.arange(shape[1]) // 37), np.arange(shape[2]) // 29)
         % 4).astype(np.uint32)
    v[rng.random(shape) < 0.002] = 0
    return np.asfortranarray(v)


# (0.001, 1, 1000): the rule sends it to the envelope; (3.3, 0.7, 29.1): digits of its own
@pytest.mark.parametrize("aniso", [(4, 4, 40), (1, 1, 1), (3.3, 0.7, 29.1), (0.001, 1, 1000)])
@pytest.mark.parametrize("kind", ["solid", "hole", "noise", "slabs"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 31, 33), (33, 32, 64), (32, 25, 97), (70, 129, 1), (5, 24, 260)])
def test_scans_match_oracle(gpu, shape, kind, aniso):
    labels = _labels(shape, kind)
    for black_border in (False, True):
        np.testing.assert_array_equal(_edt(labels, aniso, black_border), oracle.edt(labels, aniso, black_border))


@pytest.mark.parametrize("length", [1706, 1707])
@pytest.mark.parametrize("axis", [1, 2])
def test_lines_past_shared_memory(gpu, length, axis):
    """1706 voxels fit a CTA's shared memory, 1707 take the envelope, in that axis's pass alone."""
    from brook_b200 import _native as n
    from test_zz_no_alloc import _device_fortran, _edt_noalloc
    import torch

    labels = _labels((7, length, 3) if axis == 1 else (7, 3, length), "slabs")
    expected = oracle.edt(labels, (8, 8, 40), False)
    np.testing.assert_array_equal(_edt(labels, (8, 8, 40), False), expected)
    out = torch.full((labels.size,), -1.0, dtype=torch.float32, device="cuda")
    assert _edt_noalloc(_device_fortran(labels.view(np.int32)), out, (8, 8, 40), False,
                        torch.cuda.current_stream()) == n.SUCCESS
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy().reshape(labels.shape, order="F"), expected)


@pytest.mark.parametrize("length", [1706, 1707])
def test_batch_with_a_long_volume(gpu, length):
    """The distance fields of a batch, one volume of which has the longest line that scans or one too long for it."""
    from test_gpu_parity import assert_same, bk

    opts = dict(teasar_params=dict(scale=1.5, const=30, pdrf_scale=100000, pdrf_exponent=4), anisotropy=(8, 8, 40),
                dust_threshold=10)
    volumes = [_labels((12, 11, length), "slabs"), _labels((40, 33, 29), "slabs")]
    got = bk().skeletonize_batch(volumes, output="packed", **opts)
    for i, v in enumerate(volumes):
        assert_same(got[i], oracle.skeletonize(v, threads=8, **opts), str(v.shape))


def test_envelope_in_batches_of_the_fixed_scratch(gpu):
    """Spacings that the scans refuse, in a volume whose y pass needs more envelope stacks than the fixed scratch holds."""
    from brook_b200 import _native as n
    from test_zz_no_alloc import _device_fortran, _edt_noalloc
    import torch

    labels, spacing = _labels((256, 256, 64), "slabs"), (0.01, 8, 400)
    out = torch.full((labels.size,), -1.0, dtype=torch.float32, device="cuda")
    assert _edt_noalloc(_device_fortran(labels.view(np.int32)), out, spacing, False,
                        torch.cuda.current_stream()) == n.SUCCESS
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy().reshape(labels.shape, order="F"), oracle.edt(labels, spacing, False))


@pytest.mark.parametrize("wall", [None, 0, 31, 32, 33, -1])
@pytest.mark.parametrize("shape", [(97, 64, 65), (130, 95, 34), (64, 63, 160)])
def test_thick_boxes_match_oracle(gpu, shape, wall):
    """Voxels farther from the walls than the near steps, whose own block of 32 is passed over: one object with a plane of
    background across y and z (or none) beside a block's edges, at the line's first and last voxel too."""
    labels = np.ones(shape, np.uint32, order="F")
    if wall is not None:
        labels[:, wall, :] = 0
        labels[:, :, wall] = 0
    for aniso in ((1, 1, 1), (4, 3, 2)):
        for black_border in (False, True):
            np.testing.assert_array_equal(_edt(labels, aniso, black_border), oracle.edt(labels, aniso, black_border))
