"""The FP64 rerun's collision search decides as the f64 oracle's does for points
that hit a plane exactly on the edge its two triangles share.

The search takes a point as inside a face by the signs of three differences of
products; on an edge the two products are equal, and the difference is a zero
only while both are rounded the same way.  A point that both faces took as
outside would go through the plane.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fgb():
    import feriphys_gb300

    feriphys_gb300._lib()
    return feriphys_gb300


@pytest.mark.parametrize("h", [3.0, 1.0, 0.1, 1.0 / 3.0, 2.7])
def test_points_on_a_shared_edge_are_hit(fgb, orc, h):
    rng = np.random.default_rng(7)
    n = 20_000
    corners = np.array([[-h, 0, -h], [h, 0, -h], [-h, 0, h], [h, 0, h]], np.float32)
    tris = np.array([0, 2, 1, 1, 2, 3], np.uint32)  # they share the diagonal x = -z
    h32 = float(corners[3, 0])
    x = rng.uniform(-0.99 * h32, 0.99 * h32, n).astype(np.float32)
    pts = np.zeros((n, 10), np.float32)
    pts[:, 0] = 0.01
    pts[:, 1], pts[:, 2], pts[:, 3] = x, rng.uniform(1e-4, 1e-2, n), -x
    pts[:, 5] = -rng.uniform(30.0, 60.0, n)  # a step of 0.05 to 0.1 down
    pts[:, 4] = rng.uniform(-0.5, 0.5, n)    # and along the diagonal, so that the crossing point takes all of a double
    pts[:, 6] = -pts[:, 4]
    dt = 1.0 / 600.0

    g = fgb.SpringyMesh.new(pts[:, 1:4], [], 0.01 * n, 1.0, 1.0)
    g.set_precision(64)
    g.set_points(pts)
    gs = fgb.Simulation.new([g], [fgb.CollidableMesh.new(corners, tris)])
    gs.set_config(fgb.Config.make(dt=dt, gravity=(0, 0, 0), wind=(0, 0, 0), lift_coefficient=0.0, drag_coefficient=0.0,
                                  coefficient_of_restitution=0.3, coefficient_of_friction=0.2))
    gs.step(1)

    o = orc.SpringyMesh.new(pts[:, 1:4], [], 0.01 * n, 1.0, 1.0)
    o.set_points(pts)
    o = o.widen()
    os_ = orc.Simulation([o], [orc.CollidableMesh(corners, tris)])
    os_.set_config(orc.Config.make(0, dt, (0, 0, 0), (0, 0, 0), 0.0, 0.0, 0.3, 0.2))
    os_.step(1)

    got, want = g.get_points_f64(), o.get_points()
    assert (want[:, 5] > 0).all()  # every point rebounds
    assert np.array_equal(got[:, 5] > 0, want[:, 5] > 0)
    # the rerun keeps the obstacles' normals in f32 (2^-24 relative), and a response has the normal squared
    assert np.abs(got[:, 1:7] - want[:, 1:7]).max() <= 4 * 2.0 ** -24 * np.abs(want[:, 1:7]).max()
