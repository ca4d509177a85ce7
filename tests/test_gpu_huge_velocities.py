"""The tiled step where a cloth's edge meets the largest velocities and winds.

Struts and faces that a boundary tile's cloth does not have are evaluated with
zero constants against points far outside; with velocities near the largest
float such a term overflows before it is multiplied by zero.  The general
gather, which never looks at what does not exist, stays finite there, and the
tiled step has to give its bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fgb():
    import feriphys_gb300

    feriphys_gb300._lib()
    return feriphys_gb300


def _step(fgb, rows, cols, path, points, wind):
    s = 1.0 / 16
    m = fgb.Cloth.new(rows, cols, s, (0.0, 0.0, 0.0), 0.01, 500 * s, 0.5 * s, 250 * s, 0.5 * s, 50 * s, 0.5 * s,
                      [0]).mesh
    m.set_path(path)
    sim = fgb.Simulation.new([m], [])
    sim.set_config(fgb.Config.make(dt=1.0 / 6000.0, gravity=(0.0, -0.1, 0.0), wind=wind, lift_coefficient=0.0,
                                   drag_coefficient=0.0))
    m.set_points(points)
    sim.step(1)
    return m.get_points()


@pytest.mark.parametrize("rows,cols", [(2, 2), (4, 16), (8, 32), (8, 48), (300, 200)])
def test_corner_velocity(fgb, rows, cols):
    """One corner of a flat cloth moves along the cloth's normal, which no axis
    is near, so that no real strut or face of it gets a force."""
    s = np.float32(1.0 / 16)
    r, c = np.mgrid[0:rows, 0:cols].astype(np.float32)
    p = np.zeros((rows * cols, 10), np.float32)
    p[:, 0] = 0.01
    p[:, 1], p[:, 2], p[:, 3] = (s * c).ravel(), (-s * c).ravel(), (s * r).ravel()
    p[-1, 4:6] = 3.3e38
    got = [_step(fgb, rows, cols, path, p, (0.0, 0.0, 0.0)) for path in (1, 2)]
    assert np.isfinite(got[0]).all()
    assert got[0].tobytes() == got[1].tobytes()


@pytest.mark.parametrize("rows,cols", [(2, 2), (8, 48), (300, 200)])
def test_wind_across_a_flat_cloth(fgb, rows, cols):
    s = np.float32(1.0 / 16)
    r, c = np.mgrid[0:rows, 0:cols].astype(np.float32)
    p = np.zeros((rows * cols, 10), np.float32)
    p[:, 0] = 0.01
    p[:, 1], p[:, 2] = (s * c).ravel(), (-s * r).ravel()
    got = [_step(fgb, rows, cols, path, p, (0.0, 0.0, 1e37)) for path in (1, 2)]
    assert np.isfinite(got[0]).all()
    assert got[0].tobytes() == got[1].tobytes()
