"""The line-integral projector against the chords of the same rays in 64 bits,
at element grids that do not fill the kernel's tiles, voxel grids with unequal
axes, one and several projections per launch, rays along an axis, and a source
inside the phantom."""

import ctypes as C

import numpy as np
import pytest

import scenes
from ggems_b200 import abi

pytestmark = pytest.mark.gpu


def _chords(labels, mu, half, voxel, src, pixel):
    """Sum of mu x chord length along src -> pixel (FP64): chords between sorted
    plane crossings, the voxel at each chord's middle."""
    n = labels.shape[::-1]
    d = pixel - src
    t = [np.array([0.0, 1.0])]
    for a in range(3):
        if abs(d[a]) >= 1e-12:
            t.append((np.arange(n[a] + 1) * voxel[a] - half[a] - src[a]) / d[a])
    t = np.unique(np.clip(np.concatenate(t), 0.0, 1.0))
    mid = src + 0.5 * (t[1:] + t[:-1])[:, None] * d
    i = np.floor((mid + half) / voxel).astype(int)
    ok = np.all((i >= 0) & (i < n), axis=1)
    lab = labels[tuple(np.clip(i, 0, np.array(n) - 1)[:, ::-1].T)]
    return float((mu[lab] * (t[1:] - t[:-1]) * ok).sum() * np.linalg.norm(d))


def _along_a_face(src, d, half, voxel):
    """Whether the ray runs nearly along an axis and, where it is in the grid, near a
    voxel face or over one: rounding gives such a chord to either side."""
    with np.errstate(divide="ignore", invalid="ignore"):
        t = np.sort(np.array([(-half - src) / d, (half - src) / d]), axis=0)
    along = np.abs(d) < 1e-3 * np.linalg.norm(d)
    t_in, t_out = max(0.0, t[0][~along].max()), min(1.0, t[1][~along].min())
    for a in np.flatnonzero(along):
        k = (src[a] + np.array([t_in, t_out]) * d[a] + half[a]) / voxel[a]
        if np.floor(k[0]) != np.floor(k[1]) or np.any(np.abs(k - np.round(k)) < 0.05):
            return True
    return False


@pytest.mark.parametrize("elements,dims,voxel,count,inside", [
    ((1, 1), (7, 7, 7), (8.0, 6.0, 5.0), 1, False),
    ((33, 9), (31, 21, 11), (2.5, 3.0, 5.0), 1, False),
    ((33, 9), (12, 20, 7), (4.0, 3.0, 5.0), 1, False),
    ((1, 1), (5, 5, 5), (8.0, 8.0, 8.0), 3, False),
    ((64, 40), (31, 31, 31), (2.5, 2.5, 2.5), 5, False),
    ((40, 65), (16, 16, 16), (4.0, 4.0, 4.0), 2, True),
])
def test_projector_matches_chords(elements, dims, voxel, count, inside):
    from ggems_b200 import _native, scatter
    lib = scatter._lib()
    rng = np.random.default_rng(11)
    labels = rng.integers(0, 4, dims[::-1]).astype(np.uint8)
    mu = np.array([2e-5, 0.02, 0.06], np.float32)  # label 3 has no material: it adds nothing
    mu64 = np.append(mu.astype(np.float64), 0.0)
    sc = scenes.Scene()
    sc.add_voxelized(labels, voxel, 0)
    size = [160.0 / elements[0], 120.0 / elements[1], 10.0]
    dets, srcs = [], []
    for k in range(count):
        s = scenes.Scene()
        s.add_flat_detector(0, (elements[0], elements[1], 1), size, 1500.0, 1000.0, 0.01,
                            extra_rotation=(0.0, 0.0, 0.0 if k == 0 else float(0.3 + k)))
        dets.append(s.solids[0])
        m = scenes.geometry_matrix(scenes.SOURCE_AXIS, [("translation", (-1000.0, 0.0, 0.0))])
        a = np.float32(0.0 if k == 0 else 0.3 + k)
        rot = np.array([[np.cos(a), -np.sin(a), 0], [np.sin(a), np.cos(a), 0], [0, 0, 1]])
        srcs.append(np.array([1.0, -2.0, 0.5]) if inside else rot @ m[:3, 3])
    srcs = np.ascontiguousarray(np.array(srcs, np.float32))
    arr = (abi.gg_solid * count)(*dets)
    out = np.zeros((count, elements[1], elements[0], 2), np.float32)
    single = np.zeros((elements[1], elements[0]), np.float32)
    ctx = _native.Context(0)
    try:
        assert lib.gg_line_integrals_batch(ctx.handle, C.byref(sc.solids[0]), arr, abi.ptr(srcs, C.c_float), count,
                                           abi.ptr(mu, C.c_float), len(mu), abi.ptr(out, C.c_float)) == 0
        assert lib.gg_line_integrals(ctx.handle, C.byref(sc.solids[0]), C.byref(arr[0]), abi.ptr(srcs, C.c_float),
                                     abi.ptr(mu, C.c_float), len(mu), abi.ptr(single, C.c_float)) == 0
    finally:
        ctx.close()
    assert np.array_equal(single, out[0, ..., 1])
    np.testing.assert_allclose(out[..., 0], np.exp(-out[..., 1]), rtol=2e-6)
    half = np.array([sc.solids[0].obb.border_max[a] for a in range(3)])
    err, ref, along_axis = [], [], 0
    for k in range(count):
        m = np.array(list(dets[k].obb.matrix), np.float64).reshape(4, 4)
        for j in range(elements[1]):
            for i in range(elements[0]):
                c = [dets[k].obb.border_min[0] + (i + 0.5) * size[0], dets[k].obb.border_min[1] + (j + 0.5) * size[1], 0, 1]
                pixel = (m @ np.array(c))[:3]
                d = pixel - srcs[k]
                if _along_a_face(srcs[k].astype(np.float64), d, half, np.array(voxel)):
                    continue
                along_axis += k == 0 and np.min(np.abs(d)) < 1e-3 * np.linalg.norm(d)
                ref.append(_chords(labels, mu64, half, np.array(voxel), srcs[k].astype(np.float64), pixel))
                err.append(out[k, j, i, 1] - ref[-1])
    # odd voxel counts: the rays along an axis run through the voxels' middles
    assert inside or along_axis > 0 or not all(n % 2 for n in dims[1:])
    err, ref = np.array(err), np.array(ref)
    # positions along the ray round to 2^-24 of its ~1500 mm length at each of up to
    # ~100 crossings: chords off by up to ~1e-2 mm x 0.06 mm^-1, 1e-3 of the rays' ~1
    assert np.linalg.norm(err) <= 1e-4 * max(np.linalg.norm(ref), 1e-30)
    assert np.abs(err).max() <= 2e-3 * max(np.abs(ref).max(), 1e-30) if len(ref) else True
