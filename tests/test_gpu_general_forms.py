"""Every form of the general step gives the same bits (GPU tests): one thread a
vertex beyond the split kernel's sizes and the split kernel, over 16-bit words,
32-bit words and plain lists, and the FP64 step with and (path 4) without its
scratch of terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fgb():
    import feriphys_gb300

    feriphys_gb300._lib()
    return feriphys_gb300


def _mesh(rng, n_side=23):
    xs, ys = np.meshgrid(np.arange(n_side), np.arange(n_side))
    pos = np.stack([xs.ravel() * 0.05, ys.ravel() * 0.05, np.zeros(n_side * n_side)], 1)
    pos += rng.normal(0, 0.004, pos.shape)
    v = np.arange(n_side * n_side).reshape(n_side, n_side)
    a, b, c, d = (q.ravel() for q in (v[:-1, :-1], v[:-1, 1:], v[1:, :-1], v[1:, 1:]))
    turn = rng.random(len(a)) < 0.5
    idx = np.where(turn[:, None], np.stack([a, b, c, b, d, c], 1), np.stack([a, b, d, a, d, c], 1))
    return pos.astype(np.float32), idx.reshape(-1).astype(np.uint32)


def _run(fgb, pos, idx, ids, n_total, path, bits):
    """The mesh's vertices as `ids` of n_total points, the others loose; 30 steps
    onto a plane; the mesh's own points."""
    from feriphys_gb300 import workloads as W

    rng = np.random.default_rng(4)
    every = np.full((n_total, 3), 5.0, np.float32)
    every[ids] = pos
    m = fgb.SpringyMesh.new(every, ids[idx].astype(np.uint32), 0.002 * n_total, 12.0, 0.02)
    m.add_strut((int(ids[0]), int(ids[20])), 3.0, 0.01)
    m.add_pin(int(ids[7]))
    m.set_path(path)
    m.set_precision(bits)
    sim = fgb.Simulation.new([m], [fgb.CollidableMesh.new(*W.plane(0.02, 3.0))])
    sim.set_config(fgb.Config.make(**W.cloth_config(1.0 / 1200.0)))
    p = m.get_points()
    p[ids, 4:7] = rng.normal(0, 0.3, pos.shape)
    m.set_points(p)
    sim.step(30)
    out = m.get_points_f64() if bits == 64 else m.get_points()
    return np.ascontiguousarray(out[ids])


@pytest.mark.parametrize("scattered", [False, True])
@pytest.mark.parametrize("bits", [32, 64])
def test_same_bits(fgb, bits, scattered):
    rng = np.random.default_rng(3)
    pos, idx = _mesh(rng)
    got = []
    for n_total in (32_768, 32_769, 40_000):
        # scattered over all the ids, so that neighbours lie beyond the 16-bit words' reach
        ids = np.sort(rng.permutation(n_total)[:len(pos)])[rng.permutation(len(pos))] if scattered else np.arange(len(pos))
        got += [_run(fgb, pos, idx, ids, n_total, path, bits) for path in (1, 4)]
    assert np.isfinite(got[0]).all()
    for g in got[1:]:
        assert g.tobytes() == got[0].tobytes()
