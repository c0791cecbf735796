"""The transport kernel's fast forms of the voxel step against their general forms.

* quotient(): a * y refined twice with the correctly rounded reciprocal y of b
  (CPU, float arithmetic with exact fused multiply-adds) equals the correctly
  rounded a / b.
* On the GPU a launch takes the general voxel index (divisions, integer
  conversions) when one of its solids needs it, and plain table rows (one
  division per process) when a cross section is outside quotient()'s range or
  the tables are large: the same histories bit for bit as the fast forms, for
  power-of-two and other voxel sizes, with and without a dose map.
"""


import numpy as np
import pytest

import parity
import scenes

F = np.float32


def _quotient(a, b):
    """quotient() of gg_transport.cu in numpy: products and sums of a fused
    multiply-add in 64-bit mantissas, rounded once to float."""
    L = np.longdouble
    y = (F(1.0) / b).astype(F)

    def fma(p, q, r):
        return (p.astype(L) * q.astype(L) + r.astype(L)).astype(F)

    q = (a * y).astype(F)
    q = fma(fma(-q, b, a), y, q)
    return fma(fma(-q, b, a), y, q)


@pytest.mark.parametrize("seed", [1, 2])
def test_quotient_is_the_correctly_rounded_division(seed):
    rng = np.random.default_rng(seed)
    n = 1_000_000
    # -log(u) of transport: 6e-8 ... 22, cross sections and voxel sizes over many decades
    a = np.exp(rng.uniform(np.log(5.9e-8), np.log(1e4), n)).astype(F)
    b = np.exp(rng.uniform(np.log(1e-25), np.log(1e25), n)).astype(F)
    assert np.array_equal(_quotient(a, b), a / b)
    # mantissas at the ends, where a rounding error would show first
    ends = np.array([0, 1, 2, 3, 0x3FFFFF, 0x400000, 0x400001, 0x7FFFFC, 0x7FFFFD, 0x7FFFFE, 0x7FFFFF], np.uint32)
    ma = np.concatenate([ends, rng.integers(0, 1 << 23, 3000).astype(np.uint32)])
    a = (ma | np.uint32(0x3F800000)).view(F)
    b = (np.concatenate([ends, rng.integers(0, 1 << 23, 500).astype(np.uint32)]) | np.uint32(0x3F800000)).view(F)
    a, b = [x.reshape(-1).copy() for x in np.meshgrid(a, b)]
    assert np.array_equal(_quotient(a, b), a / b)
    assert np.array_equal(_quotient(-a, b), -a / b)
    assert not _quotient(np.zeros(3, F), b[:3]).any()


def _scene(n, voxel, dose, far_voxels, rows, more_materials=()):
    sc = scenes.Scene()
    tables = scenes.Tables(["Air", "Water", "Bone185"] + list(more_materials))
    if rows == "plain":
        # one value outside quotient()'s range, in bins that 120 keV photons never read
        tables.cross_sections[tables.energy_bins.size - 2] = F(1e-30)
    t = sc.add_tables(tables)
    labels = scenes.ellipsoid_phantom(n, voxel, seed=4)
    sc.add_voxelized(labels, (voxel, voxel, voxel), t, dose={"photon_tracking": True} if dose else None)
    # far off the beam: its voxel count decides the launch's voxel mode
    far = np.ones((1, 1, far_voxels), np.uint8)
    sc.add_voxelized(far, (1e-5, 1.0, 1.0), t, ops=[("translation", (0.0, 5000.0, 0.0))])
    sc.add_flat_detector(sc.add_tables(scenes.Tables(["GOS"])), (50, 40, 1), (8.0, 10.0, 10.0), 1500.0, 1000.0,
                         F(10.0) * scenes.KEV)
    return sc


@pytest.mark.gpu
@pytest.mark.parametrize("n,voxel,dose", [(33, 4.0, False), (40, 3.1, False), (40, 3.1, True), (64, 2.0, True)])
def test_fast_step_forms_match_the_general_ones(n, voxel, dose):
    from ggems_b200 import _native
    ctx = _native.Context(0)
    try:
        src = scenes.XRaySource(spectrum=scenes.synthetic_spectrum(), aperture_deg=9.0)
        runs = []
        for far, rows, extra in ((64, "fast", ()), ((1 << 22) + 1, "fast", ()), (64, "plain", ()),
                                 ((1 << 22) + 1, "plain", ()), (64, "fast", ["RibBone", "Aluminium", "Water", "Air"])):
            P, T, st = parity.run_gpu(ctx, _scene(n, voxel, dose, far, rows, extra), src, 30000)
            runs.append((P, T, st))
        P0, T0, st0 = runs[0]
        assert T0.histograms[0].sum() > 0 and T0.histograms[1].sum() > 0
        for P, T, st in runs[1:]:
            assert parity.history_agreement(P0, P)[0] == 1.0
            assert np.array_equal(st, st0)
            for a, b in zip(T0.histograms, T.histograms):
                assert np.array_equal(a, b)
            if dose:
                assert np.array_equal(T0.edep[0], T.edep[0])
                assert np.array_equal(T0.photon_tracking[0], T.photon_tracking[0])
    finally:
        ctx.close()
