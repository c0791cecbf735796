"""The meshed solid's hierarchy walk (four children a node) against the scan of
every octree node, on the GPU, where its tree has an unusual shape: one leaf,
nodes with fewer than four children, triangles on top of one another, and rays
along the boxes' faces (a pencil beam along an axis)."""

import numpy as np
import pytest

import parity
import scenes

F = np.float32


def _triangles(kind):
    from ggems_b200 import workloads
    if kind == "leaf":
        v = np.array([(60, 60, 60), (60, -60, -60), (-60, 60, -60), (-60, -60, 60)], F)
        return v[[(0, 1, 2), (0, 3, 1), (0, 2, 3), (1, 3, 2)]]
    v, f = workloads.icosphere({"few": 0, "copies": 1, "many": 4}[kind])
    t = (v * 70.0)[f].astype(F)
    return np.concatenate([t] * 3) if kind == "copies" else t


@pytest.mark.gpu
@pytest.mark.parametrize("kind,aperture", [("leaf", 4.0), ("few", 4.0), ("copies", 4.0), ("many", 4.0), ("many", 0.0),
                                           ("few", 0.0)])
def test_walk_matches_the_scan(tmp_path, monkeypatch, kind, aperture):
    from ggems_b200 import _native, workloads
    path = str(tmp_path / "body.stl")
    workloads.write_stl(path, _triangles(kind))
    sc = scenes.Scene()
    sc.add_meshed(path, sc.add_tables(scenes.Tables(["Water"])), depth=3, dose={"dosel_size": (10.0, 10.0, 10.0)})
    # off the axis: a ray through shared vertices and edges counts what rounding makes of it, in either order
    src = scenes.XRaySource(spectrum=scenes.synthetic_spectrum(), aperture_deg=aperture, focal=(0.0, 20.0, 20.0))
    ctx = _native.Context(0)
    try:
        runs = []
        for bvh in ("0", "1"):
            monkeypatch.setenv("GGEMS_B200_MESH_BVH", bvh)
            runs.append(parity.run_gpu(ctx, sc, src, 50000))
    finally:
        ctx.close()
    (P0, T0, s0), (P1, T1, s1) = runs
    assert T0.hit[0].sum() > 1000
    assert parity.history_agreement(P1, P0, pos_tol=1e-2)[0] > 0.999
    assert (s0 == s1).all(0).mean() > 0.9999
    assert abs(T1.edep[0].sum() - T0.edep[0].sum()) <= 0.002 * T0.edep[0].sum()
