"""The transport kernel's short voxel step against its general forms.

* surely_crosses() (CPU, float arithmetic): where it says that a photon crosses
  its voxel, no process's -logf(u) / sigma is below the distance, with the
  logarithm an ulp either way.
* On the GPU a launch takes the general index, clamp and distance when a grid of
  it is too long for the short ones: the same histories, states and tallies bit
  for bit as with both short forms of the index, for odd voxel counts, voxel sizes
  with and without a power of two, a rotated phantom, a pencil beam along each axis
  of the grid, and with the track-length estimator.
"""

import math

import numpy as np
import pytest

import parity
import scenes

F = np.float32


def _fma(a, b, c):
    return (a.astype(np.longdouble) * b.astype(np.longdouble) + c.astype(np.longdouble)).astype(F)


@pytest.mark.parametrize("seed", [1, 2])
def test_a_sure_crossing_has_no_nearer_interaction(seed):
    rng = np.random.default_rng(seed)
    n = 2_000_000
    sigma = np.exp(rng.uniform(np.log(1e-12), np.log(1e3), n)).astype(F)
    distance = np.exp(rng.uniform(np.log(5e-4), np.log(3e3), n)).astype(F)
    draw = rng.integers(0, 1 << 32, n, dtype=np.uint64)
    # half of the draws where the test's two sides meet
    edge = (1.0 - sigma.astype(np.float64) * distance) * 2.0 ** 32 * (1.0 + rng.normal(0, 1e-6, n))
    pick = (rng.random(n) < 0.5) & (edge > 0) & (edge < 2.0 ** 32)
    draw[pick] = edge[pick].astype(np.uint64)
    draw[:64] = np.arange(64)
    draw[64:128] = (1 << 32) - 1 - np.arange(64)
    x = draw.astype(np.uint32).astype(F)
    reach = (distance * F(float.fromhex("0x1.00004p+32"))).astype(F)
    sure = _fma(sigma, reach, x) < F(2.0 ** 32 - 2.0 ** 11)
    assert 0.2 < sure.mean() < 0.9 and (sure & pick).any() and (~sure & pick).any()
    u = _fma(x, np.full(n, float.fromhex("-0x1.ffp-56"), F), (x * F(2.0 ** -32)).astype(F))
    with np.errstate(divide="ignore"):
        log = (-np.log(u.astype(np.float64))).astype(F)
    for a in (log, np.nextafter(log, F(0)), np.nextafter(log, F(np.inf))):
        assert ((a / sigma)[sure] >= distance[sure]).all()


# A solid far off the beam that decides the launch's form of the voxel step
# (voxel size in mm along x, voxels): short with powers of two, short with
# reciprocals, general (longer than the 2048 mm that the short forms take).
FAR = {"pow2": (0.015625, 64), "reciprocal": (0.02, 64), "general": (0.02, 1 << 17)}


def _forms(voxel):
    """The forms that a grid of these voxels can be stepped through with."""
    assert all((size * count > 2048.0) == (form == "general") and size > 0.008 for form, (size, count) in FAR.items())
    assert all((math.frexp(size)[0] == 0.5) == (form == "pow2") for form, (size, _) in FAR.items())
    return ["pow2"] * (math.frexp(voxel)[0] == 0.5) + ["reciprocal", "general"]


def _scene(n, voxel, ops, dose, form, tle=False):
    sc = scenes.Scene()
    t = sc.add_tables(scenes.Tables(["Air", "Water", "Bone185"]))
    sc.add_voxelized(scenes.ellipsoid_phantom(n, voxel, seed=4), (voxel, voxel, voxel), t, ops=ops,
                     dose={"photon_tracking": True, "tle": tle} if dose else None)
    size, count = FAR[form]
    sc.add_voxelized(np.ones((1, 1, count), np.uint8), (size, 1.0, 1.0), t, ops=[("translation", (0.0, 5000.0, 0.0))])
    sc.add_flat_detector(sc.add_tables(scenes.Tables(["GOS"])), (50, 40, 1), (8.0, 10.0, 10.0), 1500.0, 1000.0,
                         F(10.0) * scenes.KEV)
    return sc


@pytest.mark.gpu
@pytest.mark.parametrize("n,voxel,rotation,dose,aperture", [
    (33, 4.0, (0.0, 0.0, 0.0), False, 9.0),
    (40, 3.1, (0.0, 0.0, 0.0), False, 9.0),
    (64, 2.0, (0.0, 0.0, 0.0), True, 9.0),
    (64, 2.0, (0.0, 0.0, 0.0), "tle", 9.0),
    (41, 3.1, (0.0, 0.0, 0.3), True, 9.0),
    (41, 3.1, (0.0, 0.0, 0.3), "tle", 9.0),
    (117, 0.7, (0.2, 0.1, 0.0), False, 4.0),
    (40, 2.5, (0.0, 0.0, 0.0), True, 0.0),
    (40, 2.5, (0.0, 0.0, math.pi / 2), True, 0.0),
    (40, 2.5, (0.0, math.pi / 2, 0.0), False, 0.0),
    (1, 60.0, (0.0, 0.0, 0.0), True, 2.0),
    (1, 64.0, (0.0, 0.0, 0.0), "tle", 2.0),
])
def test_short_steps_match_the_general_forms(n, voxel, rotation, dose, aperture):
    from ggems_b200 import _native
    ctx = _native.Context(0)
    try:
        src = scenes.XRaySource(spectrum=scenes.synthetic_spectrum(), aperture_deg=aperture)
        runs = [parity.run_gpu(ctx, _scene(n, voxel, [("rotation", rotation)], dose, form, dose == "tle"), src, 40000)
                for form in _forms(voxel)]
        P0, T0, st0 = runs[0]
        assert T0.histograms[0].sum() > 0
        if dose:
            assert T0.hit[0].sum() > 0
        for P1, T1, st1 in runs[1:]:
            assert parity.history_agreement(P0, P1)[0] == 1.0
            assert np.array_equal(st0, st1)
            for a, b in zip(T0.histograms, T1.histograms):
                assert np.array_equal(a, b)
            if dose:
                for name in ("edep", "hit", "photon_tracking"):
                    assert np.array_equal(getattr(T0, name)[0], getattr(T1, name)[0])
                # a sum of doubles in any order: n terms, each within (n - 1) 2^-53 of the sum, n <= the hits
                e = T0.edep_squared[0]
                assert (np.abs(T1.edep_squared[0] - e) <= np.maximum(T0.hit[0], 1) * 2.0 ** -52 * e).all()
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("beside", ["world", "mesh", "no stash", "stash of 64 registers"])
def test_other_kernels_of_the_general_forms(tmp_path, beside):
    """The forms again in the kernels for a world grid, for a meshed solid and for other stashes."""
    from ggems_b200 import _native, workloads
    ctx = _native.Context(0)
    try:
        if "stash" in beside:
            ctx.set_stash(registers=0 if beside == "no stash" else 64)
        src = scenes.XRaySource(spectrum=scenes.synthetic_spectrum(), aperture_deg=6.0)
        runs = []
        for form in FAR:
            sc = _scene(32, 4.0, [], True, form)
            if beside == "world":
                sc.set_world((20, 20, 20), (100.0, 100.0, 100.0))
            if beside == "mesh":
                path = str(tmp_path / "ball.stl")
                v, f = workloads.icosphere(2)
                workloads.write_stl(path, (v * 40.0)[f].astype(F))
                sc.add_meshed(path, sc.add_tables(scenes.Tables(["Water"])), depth=3,
                              ops=[("translation", (-300.0, 0.0, 0.0))], dose={"dosel_size": (10.0, 10.0, 10.0)})
            runs.append(parity.run_gpu(ctx, sc, src, 40000))
        P0, T0, st0 = runs[0]
        assert T0.hit[0].sum() > 1000 and (beside != "mesh" or T0.hit[1].sum() > 1000)
        for P1, T1, st1 in runs[1:]:
            assert parity.history_agreement(P0, P1)[0] == 1.0 and np.array_equal(st0, st1)
            for a, b in zip(T0.histograms + T0.edep + T0.hit, T1.histograms + T1.edep + T1.hit):
                assert np.array_equal(a, b)
            if beside == "world":
                assert T0.world["photon_tracking"].sum() > 0
                for name in ("photon_tracking", "energy", "momentum_x", "momentum_y", "momentum_z"):
                    assert np.array_equal(T0.world[name], T1.world[name])
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("value,count", [(float("nan"), 1), (float("inf"), 7), (-1.0e-30, -3)])
def test_a_detector_box_has_no_voxels(value, count):
    """gg_solid's voxel fields are a voxelized solid's: whatever a box holds there changes nothing."""
    from ggems_b200 import _native
    ctx = _native.Context(0)
    try:
        src = scenes.XRaySource(spectrum=scenes.synthetic_spectrum(), aperture_deg=9.0)
        runs = []
        for fill in (False, True):
            sc = _scene(16, 8.0, [], False, "pow2")
            if fill:
                box = sc.solids[-1]
                box.voxel_sizes[:] = [value] * 3
                box.number_of_voxels[:] = [count] * 3
            runs.append(parity.run_gpu(ctx, sc, src, 40000))
        (P0, T0, st0), (P1, T1, st1) = runs
        assert T0.histograms[0].sum() > 10000 and parity.history_agreement(P0, P1)[0] == 1.0
        assert np.array_equal(st0, st1)
        for a, b in zip(T0.histograms, T1.histograms):
            assert np.array_equal(a, b)
    finally:
        ctx.close()
