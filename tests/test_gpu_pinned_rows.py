"""Small reads into pageable memory go through pinned rows that all meshes share
(capi.cu: RowPool): reading many meshes back pins little, reads of several
threads do not mix, and the rows outlive the mesh that first used them."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fgb():
    import feriphys_gb300

    feriphys_gb300._lib()
    return feriphys_gb300


def _meshes(fgb, n, points=5):
    rng = np.random.default_rng(n)
    pos = rng.normal(0, 1, (n, points, 3)).astype(np.float32)
    meshes = [fgb.SpringyMesh.new(p, [], 0.01 * points, 1.0, 1.0) for p in pos]
    sim = fgb.Simulation.new(meshes, [])
    sim.step(0)
    return pos, meshes, sim


def _resident_kb():
    return next(int(line.split()[1]) for line in open("/proc/self/status") if line.startswith("VmRSS"))


def test_many_meshes_pin_little(fgb):
    """512 meshes with rows of their own pinned 512 x 64 KB."""
    pos, meshes, _sim = _meshes(fgb, 512)
    meshes[0].get_points()
    before = _resident_kb()
    for p, m in zip(pos, meshes):
        assert np.array_equal(m.get_points()[:, 1:4], p)
    assert _resident_kb() - before < 8 * 1024


def test_threads_do_not_mix(fgb):
    pos, meshes, _sim = _meshes(fgb, 24, points=1500)
    wrong = []

    def read(k):
        for _ in range(40):
            for j in (k, k + 12):
                if not np.array_equal(meshes[j].get_points()[:, 1:4], pos[j]):
                    wrong.append(j)

    threads = [threading.Thread(target=read, args=(k,)) for k in range(12)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_meshes_come_and_go(fgb):
    for _ in range(3):
        pos, meshes, sim = _meshes(fgb, 3)
        keep = meshes[2]
        meshes[0].get_points()
        sim = meshes = None  # noqa: F841
        assert np.array_equal(keep.get_points()[:, 1:4], pos[2])
