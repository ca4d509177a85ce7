"""Faces whose corners are exactly collinear, along no axis (GPU tests).

Their cross product is a zero only while both products of each component are
rounded; the reference then normalises a zero vector, and the face's points go
non-finite (springy_mesh.rs:629-654).  Every step form has to do so at the same
points as the oracle, raise its flag, and leave the other points alone.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PER_STEP_TOL = 1e-5  # f32, one step, with drag and lift (tests/test_gpu_parity.py)


@pytest.fixture(scope="module")
def fgb():
    import feriphys_gb300

    feriphys_gb300._lib()
    return feriphys_gb300


@pytest.fixture(scope="module")
def W():
    from feriphys_gb300 import workloads

    return workloads


def _oracle_step(orc, m, cfg):
    sim = orc.Simulation([m], [])
    sim.set_config(orc.Config.make(cfg["integration"], cfg["dt"], cfg["gravity"], cfg["wind"], cfg["lift_coefficient"],
                                   cfg["drag_coefficient"], cfg["coefficient_of_restitution"],
                                   cfg["coefficient_of_friction"]))
    sim.step(1)
    return m.get_points()[:, 1:7].astype(np.float64)


def _step(fgb, m, cfg):
    sim = fgb.Simulation.new([m], [])
    sim.set_config(fgb.Config.make(**cfg))
    sim.step(1)
    flagged = sim.synchronize()
    return m.get_points()[:, 1:7].astype(np.float64), flagged


def _compare(got, flagged, want, expect_bad):
    bad = ~np.isfinite(want).all(1)
    assert bad[expect_bad].all() and not bad.all()
    assert np.array_equal(~np.isfinite(got).all(1), bad)
    assert flagged
    ok = ~bad
    assert np.abs(got[ok] - want[ok]).max() <= PER_STEP_TOL * np.abs(want[ok]).max()


# points: enough for the split general kernel, and one more than it takes
@pytest.mark.parametrize("bits,n_total", [(32, 3000), (32, 32_769), (64, 3000)])
def test_general_mesh(fgb, orc, W, bits, n_total):
    rng = np.random.default_rng(1)
    n_faces = 900
    corners = rng.normal(0, 0.1, (n_faces, 3, 3)).astype(np.float32)
    line = np.arange(n_faces) % 2 == 0
    e = rng.normal(0, 0.1, (n_faces, 3)).astype(np.float32)
    for k in np.flatnonzero(line):  # -e, 0, e: every edge exact; any corner first
        corners[k] = np.roll(np.stack([-e[k], 0 * e[k], e[k]]), k // 2, 0)
    pos = rng.normal(0, 1, (n_total, 3)).astype(np.float32)
    pos[:3 * n_faces] = corners.reshape(-1, 3)
    idx = np.arange(3 * n_faces, dtype=np.uint32)
    cfg = W.cloth_config(1.0 / 6000.0)
    g = fgb.SpringyMesh.new(pos, idx, 0.01 * n_total, 5.0, 0.01)
    o = orc.SpringyMesh.new(pos, idx, 0.01 * n_total, 5.0, 0.01)
    if bits == 64:
        g.set_precision(64)
        o = o.widen()
    got, flagged = _step(fgb, g, cfg)
    _compare(got, flagged, _oracle_step(orc, o, cfg), np.flatnonzero(np.repeat(line, 3)))


@pytest.mark.parametrize("path", [1, 2, 3])
@pytest.mark.parametrize("rows,cols", [(9, 12), (60, 130)])
def test_cloth(fgb, orc, W, rows, cols, path):
    s = 0.05
    args = (rows, cols, s, (0.0, 0.0, 0.0), 0.01, 500 * s, 0.5 * s, 250 * s, 0.5 * s, 50 * s, 0.5 * s)
    g, o = fgb.Cloth.new(*args, [0]).mesh, orc.SpringyMesh.cloth(*args, pinned=[0])
    g.set_path(path)
    rng = np.random.default_rng(rows)
    p = o.get_points()
    p[:, 1:4] += rng.normal(0, 2e-3, (rows * cols, 3)).astype(np.float32)
    q = p.reshape(rows, cols, 10)
    bad = []
    for r in range(1, rows - 2, 4):
        for c in range(1, cols - 2, 5):
            e = rng.normal(0, 0.05, 3).astype(np.float32)
            face = [(r, c + 1), (r + 1, c), (r, c)] if (r + c) % 2 else [(r, c + 1), (r + 1, c + 1), (r + 1, c)]
            for k, (a, b) in enumerate(face):
                q[a, b, 1:4] = (k - 1) * e
                bad.append(a * cols + b)
    g.set_points(p)
    o.set_points(p)
    cfg = W.cloth_config(1.0 / 6000.0)
    got, flagged = _step(fgb, g, cfg)
    _compare(got, flagged, _oracle_step(orc, o, cfg), np.array(bad))


KERNEL = r"""
#include "devmath.cuh"
using namespace fgb;
__global__ void crosses(const double* ab, int n, double* out) {  // n pairs of vectors -> unfused, fused, the normal's
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* q = ab + 6 * i;
  const V3<double> a{q[0], q[1], q[2]}, b{q[3], q[4], q[5]};
  const V3<double> r[3] = {cross(a, b), face_cross(a, b), normal_cross(a, b)};
  for (int k = 0; k < 3; ++k) {
    out[9 * i + 3 * k] = r[k].x;
    out[9 * i + 3 * k + 1] = r[k].y;
    out[9 * i + 3 * k + 2] = r[k].z;
  }
}
extern "C" int run_crosses(const double* ab, int n, double* out) {
  double *d, *o;
  if (cudaMalloc(&d, n * 48) != cudaSuccess || cudaMalloc(&o, n * 72) != cudaSuccess) return -1;
  cudaMemcpy(d, ab, n * 48, cudaMemcpyHostToDevice);
  crosses<<<(n + 127) / 128, 128>>>(d, n, o);
  const cudaError_t e = cudaMemcpy(out, o, n * 72, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(o);
  return e == cudaSuccess ? 0 : -2;
}
"""


def test_normal_cross_is_zero_where_the_unfused_one_is(tmp_path):
    """FP64 edges with all their bits: exactly collinear ones, ones that are a
    rounding away from it, and any, at magnitudes up to the ends of the range."""
    src, lib = str(tmp_path / "cross.cu"), str(tmp_path / "libcross.so")
    open(src, "w").write(KERNEL)
    subprocess.check_call(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-fmad=false",
                           "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(ROOT, "feriphys_gb300", "csrc"),
                           "-o", lib, src])
    rng = np.random.default_rng(2)
    n = 60_000
    a = rng.normal(0, 1, (n, 3)) * 2.0 ** rng.choice([-520, -500, -480, -60, 0, 60, 480], (n, 1))
    a[rng.random((n, 3)) < 0.1] = 0.0
    b = a * rng.choice([2.0, -1.0, -0.5, 1.0, 3.0, 1.0 / 3.0, 0.7], (n, 1))  # the first four exact
    b[-20_000:] += rng.normal(0, 1, (20_000, 3)) * np.abs(a[-20_000:]) * 2.0 ** rng.integers(-60, 0, (20_000, 1))
    ab = np.ascontiguousarray(np.concatenate([a, b], 1))
    out = np.zeros((n, 3, 3))
    l = C.CDLL(lib)
    l.run_crosses.argtypes = [C.c_void_p, C.c_int, C.c_void_p]
    assert l.run_crosses(ab.ctypes.data, n, out.ctypes.data) == 0
    unfused, fused, normal = out[:, 0], out[:, 1], out[:, 2]
    zero = (unfused == 0).all(1)
    assert zero.sum() > 20_000 and ((fused != 0).any(1) & zero).sum() > 10_000
    assert np.array_equal((normal == 0).all(1), zero)
    of = [(normal.view(np.uint64) == x.view(np.uint64)).all(1) for x in (unfused, fused)]
    assert (of[0] | of[1]).all()
    far = np.abs(fused).max(1) > 1e-12 * np.abs(a).max(1) * np.abs(b).max(1)
    assert of[1][far & (np.abs(a).max(1) > 2.0 ** -400)].all()
