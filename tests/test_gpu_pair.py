"""The tiled kernel's packed arithmetic and its rare branches on the GPU.

* pair.cuh: the root of two lanes is the IEEE square root, and the reciprocal
  of such a root the IEEE reciprocal, for every float in the stated range and,
  for the form that also takes zeros, for zero.
* The tiled kernel gives the bits of the general gather where its terms leave
  the fast range (coincident points at the cloth's edges, no wind on a flat
  cloth, extreme and non-finite coordinates), with carried forces, with the
  reference's RK4, and with more obstacles than have a box of their own.
"""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

KERNEL = r"""
#include "pair.cuh"
using namespace fgb;
__global__ void roots(unsigned long long* bad) {
  unsigned long long b[3] = {0, 0, 0};
  for (unsigned long long i = kRootLo + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
       i <= kRootLo + (unsigned long long)kRootSpan; i += (unsigned long long)gridDim.x * blockDim.x) {
    const float x = __uint_as_float(unsigned(i)), x2 = __uint_as_float(unsigned(i) ^ 1u);
    const float r = __fsqrt_rn(x), r2 = __fsqrt_rn(x2);
    const float2 s = upk(root_fast2(pk(x, x2)));
    if (s.x != r || s.y != r2) ++b[0];
    const float2 q = upk(rcp_root_fast2(pk(r, r2)));
    if (q.x != __fdiv_rn(1.0f, r) || q.y != __fdiv_rn(1.0f, r2)) ++b[1];
    uint32_t far = 0;
    const float2 z = upk(root_or_zero<true>(pk(x, 0.0f), far));
    if (z.x != r || __float_as_uint(z.y) != 0u || far > kRootSpan) ++b[2];
  }
  for (int j = 0; j < 3; ++j)
    if (b[j]) atomicAdd(bad + j, b[j]);
}
extern "C" int run_roots(unsigned long long* out) {
  unsigned long long* d;
  if (cudaMalloc(&d, 24) != cudaSuccess) return -1;
  cudaMemset(d, 0, 24);
  roots<<<4096, 256>>>(d);
  if (cudaMemcpy(out, d, 24, cudaMemcpyDeviceToHost) != cudaSuccess) return -2;
  cudaFree(d);
  return 0;
}
"""


@pytest.fixture(scope="module")
def fgb():
    import feriphys_gb300

    feriphys_gb300._lib()
    return feriphys_gb300


def test_roots_exact():
    d = tempfile.mkdtemp(prefix="fgb_pair_")
    src, lib = os.path.join(d, "pair.cu"), os.path.join(d, "libpair.so")
    open(src, "w").write(KERNEL)
    subprocess.check_call(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-fmad=false",
                           "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(ROOT, "feriphys_gb300", "csrc"),
                           "-o", lib, src])
    l = C.CDLL(lib)
    out = (C.c_ulonglong * 3)()
    assert l.run_roots(out) == 0
    assert list(out) == [0, 0, 0]


def _run(fgb, W, path, rows, cols, edit, steps=3, rk4=False, wind=(2.0, 0.0, 1.0), obstacles=None, force=False):
    s = 1.0 / 31
    lt, ls, lb = s, s * 2 ** 0.5, 2 * s
    args = (rows, cols, s, (0.0, 0.0, 0.0), 0.01, 500 * lt, 0.5 * lt, 250 * ls, 0.5 * ls, 50 * lb, 0.5 * lb)
    mesh = fgb.Cloth.new(*args, [0]).mesh
    mesh.set_path(path)
    obs = [W.plane(-0.3)] if obstacles is None else obstacles
    sim = fgb.Simulation.new([mesh], [fgb.CollidableMesh.new(*o) for o in obs])
    cfg = W.cloth_config(1.0 / 6000.0, 1 if rk4 else 0)
    cfg["wind"] = wind
    sim.set_config(fgb.Config.make(**cfg))
    p = mesh.get_points()
    edit(p.reshape(rows, cols, 10))
    if force:
        p[:, 7:10] = np.random.default_rng(1).normal(0, 0.01, (rows * cols, 3))
    sim.step(0)
    mesh.set_points(p)  # on the device already: the forces are carried into the first step
    sim.step(steps)
    return np.ascontiguousarray(mesh.get_points())


def _same(a, b):
    """Bit for bit, every NaN equal to every other."""
    nan = np.isnan(a) & np.isnan(b)
    return ((a.view(np.uint32) == b.view(np.uint32)) | nan).all()


def _jitter(q):
    q[..., 1:7] += np.random.default_rng(q.size).normal(0, 2e-3, q[..., 1:7].shape).astype(np.float32)


def _coincident(q):
    q[-1, :, 1:4] = q[-2, :, 1:4]  # the last two rows, which own no binding struts, on top of each other
    q[:, -1, 1:4] = q[:, max(q.shape[1] - 3, 0), 1:4]
    q[0, 0, 1:4] = q[0, 1, 1:4]


def _far_away(q):
    q[..., 1:4] *= np.float32(2.0 ** 62)


def _huge_row(q):
    _jitter(q)
    q[q.shape[0] // 2, :, 1:4] *= np.float32(1e30)


def _broken(q):
    _jitter(q)
    q[1, 1, 1] = np.nan
    q[-1, -1, 2] = np.inf
    q[0, -1, 4] = np.inf


CASES = {"jitter": _jitter, "flat": lambda q: None, "coincident": _coincident, "far_away": _far_away,
         "huge_row": _huge_row, "broken": _broken}


@pytest.mark.parametrize("rows,cols", [(2, 2), (5, 16), (9, 33), (20, 50), (40, 170)])
@pytest.mark.parametrize("case", sorted(CASES))
def test_tiled_equals_general(fgb, case, rows, cols):
    from feriphys_gb300 import workloads as W

    for rk4, wind in ((False, (2.0, 0.0, 1.0)), (True, (0.0, 0.0, 0.0)), (False, (0.0, 0.0, 3.0))):
        a, b = (_run(fgb, W, p, rows, cols, CASES[case], rk4=rk4, wind=wind) for p in (1, 2))
        assert _same(a, b), (rk4, wind)


@pytest.mark.parametrize("rows,cols", [(8, 32), (70, 95), (300, 200)])
def test_carried_forces_and_many_obstacles(fgb, rows, cols):
    """Sizes on both sides of the tile-height rule; five spheres through the cloth and a plane under it."""
    from feriphys_gb300 import workloads as W

    x, y = cols / 62.0, rows / 62.0
    obs = [W.plane(-0.8 * y)] + [W.uv_sphere((a * x, b * y, 0.01), 0.2 * min(x, y), 12, 8)
                                 for a, b in ((0, 0), (0.6, 0.5), (-0.6, 0.5), (0.6, -0.5), (-0.6, -0.5))]

    def edit(q):
        _jitter(q)
        q[..., 6] += np.random.default_rng(3).normal(0, 20.0, q[..., 6].shape).astype(np.float32)

    a, b = (_run(fgb, W, p, rows, cols, edit, steps=20, obstacles=obs, force=True) for p in (1, 2))
    assert np.isfinite(a).all() and _same(a, b)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("valence", [3, 6, 7, 13, 40])
def test_split_step_any_valence(fgb, orc, bits, valence):
    """A fan around one vertex of the given valence beside a strip, in a mesh
    small enough for the split general step (several rounds of face shares for
    the hub, none for a loose point), against the oracle."""
    rng = np.random.default_rng(valence)
    a = np.linspace(0, 2 * np.pi, valence, endpoint=False)
    ring = np.stack([np.cos(a), np.sin(a), 0.1 * np.cos(3 * a)], 1)
    extra = rng.normal(0, 1, (9, 3)) + 3.0
    pos = np.concatenate([[[0, 0, 0.2]], ring, extra]).astype(np.float32)
    idx = [x for k in range(valence) for x in (0, 1 + k, 1 + (k + 1) % valence)]
    b = 1 + valence
    idx += [x for k in range(6) for x in (b + k, b + k + 1, b + k + 2)]  # leaves the last point loose
    m = fgb.SpringyMesh.new(pos, idx, 0.01 * len(pos), 5.0, 0.01)
    m.add_pins([b])
    m.set_precision(bits)
    cfg = dict(dt=1.0 / 6000.0, gravity=(0.0, -0.1, 0.0), wind=(2.0, 0.5, 1.0))
    sim = fgb.Simulation.new([m], [])
    sim.set_config(fgb.Config.make(lift_coefficient=0.3, drag_coefficient=0.6, coefficient_of_restitution=0.3,
                                   coefficient_of_friction=0.2, **cfg))
    om = orc.SpringyMesh.new(pos, np.array(idx, np.uint32), 0.01 * len(pos), 5.0, 0.01)
    om.add_pins(np.array([b], np.uint32))
    osim = orc.Simulation([om], [])
    osim.set_config(orc.Config.make(0, cfg["dt"], cfg["gravity"], cfg["wind"], 0.3, 0.6, 0.3, 0.2))
    for _ in range(5):
        sim.step(1)
        osim.step(1)
    g, o = m.get_points()[:, 1:7].astype(np.float64), om.get_points()[:, 1:7].astype(np.float64)
    assert np.abs(g - o).max() / np.abs(o).max() <= 1e-6  # five steps of f32 rounding; the terms are O(1) of the state


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 1000])
def test_exchange_at_any_offset(fgb, n, offset, pinned):
    """Stateful rows from and to a buffer at every alignment a float array can
    have, at the edges of the conversion's 256-point blocks, unchanged."""
    import torch

    rng = np.random.default_rng(n + offset)
    m = fgb.SpringyMesh.new(rng.normal(0, 1, (n, 3)).astype(np.float32), [], 0.01 * n, 1.0, 1.0)
    sim = fgb.Simulation.new([m], [])
    sim.step(0)
    flat = lambda: torch.zeros(10 * n + offset, pin_memory=pinned).numpy()[offset:].reshape(n, 10)  # noqa: E731
    src, dst = flat(), flat()
    src[:] = rng.normal(0, 1, (n, 10)).astype(np.float32)
    m.set_points(src)
    got = m.get_points(dst)
    assert got.tobytes() == src.tobytes()


@pytest.mark.parametrize("steps", [1, 8, 9, 25, 70])
def test_checked_steps_launched_ahead(fgb, steps):
    """The checked rollout launches runs of 8, 16, 32 coarse steps ahead of
    their verdicts, and single ones after a failure: whether no step fails,
    some do (at the ends of runs and inside them) or all do, the counts and
    the states are those of the loop that waits for each verdict."""
    from feriphys_gb300 import workloads as W

    batch = W.c2(n_cloths=3, lo=6, hi=40, seed=2, dt=1.0 / 6000.0)
    sur = fgb.Surrogate.new(21)
    chk = fgb.SurrogateCheck.make(energy_growth=1e-3, energy_abs=1e-7, max_strain=0.5)
    counts = []
    for scale in (1e-4, *np.geomspace(1e-2, 1e-1, 7), 100.0):
        sur.set_normalization(np.zeros(54), np.ones(54), np.zeros(3), np.full(3, scale))
        got = []
        for ahead in (True, False):
            sim, meshes, _ = W.build_batch(batch, fgb)
            sim.set_graphs(ahead)
            got.append((sim.step_surrogate(sur, 3, steps, chk), [m.get_points() for m in meshes]))
        assert got[0][0] == got[1][0], scale
        for a, b in zip(got[0][1], got[1][1]):
            assert np.array_equal(a, b), scale
        counts.append(got[0][0])
    assert len(set(counts)) > 1, counts


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n", [1, 1638, 1639, 5461, 5462])
def test_reads_into_pageable_and_pinned_memory(fgb, n, bits):
    """Rows read into pageable memory (through the mesh's own pinned rows up to
    64 KB: 1,638 points, or 5,461 positions) and into pinned memory are the
    same bytes."""
    import torch

    rng = np.random.default_rng(n)
    m = fgb.SpringyMesh.new(rng.normal(0, 1, (n, 3)).astype(np.float32), [], 0.01 * n, 1.0, 1.0)
    m.set_precision(bits)
    sim = fgb.Simulation.new([m], [])
    sim.step(2)
    pinned = lambda k: torch.zeros((n, k), pin_memory=True).numpy()  # noqa: E731
    for _ in range(2):
        sim.step(1)
        assert m.get_points().tobytes() == m.get_points(pinned(10)).tobytes()
        odd = np.zeros(3 * n + 1, np.float32)[1:].reshape(n, 3)
        assert m.get_positions(odd).tobytes() == m.get_positions(pinned(3)).tobytes()
        assert odd.tobytes() == m.get_points()[:, 1:4].tobytes()


@pytest.mark.parametrize("rows, cols, cloths", [(64, 64, 5), (64, 64, 10), (64, 64, 20), (61, 67, 21), (9, 9, 160)])
def test_coarse_step_is_the_same_in_any_company(fgb, rows, cols, cloths):
    """A coarse step of a cloth gives the same bits alone (a tile an SM) and
    among copies of itself, where its tiles fall to the second, third and
    fourth group of an SM, to groups that start late and to later rounds; the
    last tile of a cloth may be partly empty."""
    s = 0.02
    rng = np.random.default_rng(rows + cloths)
    kick = rng.normal(0, 0.3, (rows * cols, 3)).astype(np.float32)

    def sim_of(k):
        meshes = []
        for _ in range(k):
            m = fgb.Cloth.new(rows, cols, s, (0.0, 0.0, 0.0), 0.01, 500.0 * s, 0.5 * s, 250.0 * s, 0.5 * s, 50.0 * s,
                              0.5 * s, np.asarray([0], np.uint32)).mesh
            pts = m.get_points()
            pts[:, 4:7] = kick
            m.set_points(pts)
            meshes.append(m)
        sim = fgb.Simulation.new(meshes, [])
        sim.set_config(fgb.Config.make(dt=1.0 / 6000.0, gravity=(0.0, -9.8, 0.0), wind=(1.0, 0.5, 0.2)))
        return sim, meshes

    sur = fgb.Surrogate.new(3)
    sur.set_normalization(np.zeros(54), np.ones(54), np.zeros(3), np.full(3, 0.05))
    one, (alone,) = sim_of(1)
    many, meshes = sim_of(cloths)
    assert one.step_surrogate(sur, 10, 3) == 0 and many.step_surrogate(sur, 10, 3) == 0
    want = alone.get_points()
    assert np.isfinite(want).all() and not np.array_equal(want[:, 4:7], kick)
    for m in meshes:
        assert m.get_points().tobytes() == want.tobytes()


@pytest.mark.parametrize("integration", [0, 1])
@pytest.mark.parametrize("rows, cols, faces", [(1, 2, True), (2, 2, True), (5, 7, True), (9, 9, False), (33, 31, True),
                                               (190, 180, True)])
def test_f64_step_is_its_phases(fgb, rows, cols, faces, integration):
    """The FP64 step (terms once each, then per vertex) gives the bits of its
    phases called one by one (accumulate_forces sums vertex by vertex), for
    loose points, few and many faces, struts without faces, pins, carried
    forces and an obstacle."""
    from feriphys_gb300 import workloads as W

    rng = np.random.default_rng(rows + 10 * cols)
    y, x = np.mgrid[0:rows, 0:cols]
    pos = np.stack([x * 0.1, 0.02 * rng.normal(0, 1, x.shape), y * 0.1], -1).reshape(-1, 3).astype(np.float32)
    v = np.arange(rows * cols).reshape(rows, cols)
    a, b, c, d = (q.reshape(-1) for q in (v[:-1, :-1], v[:-1, 1:], v[1:, :-1], v[1:, 1:]))
    idx = np.stack([a, b, c, b, d, c], 1).reshape(-1).astype(np.uint32) if faces else np.zeros(0, np.uint32)
    cfg = fgb.Config.make(integration=integration, dt=1.0 / 2000.0, gravity=(0.0, -0.1, 0.0), wind=(2.0, 0.5, 1.0),
                          lift_coefficient=0.3, drag_coefficient=0.6, coefficient_of_restitution=0.3,
                          coefficient_of_friction=0.2)
    obstacle = fgb.CollidableMesh.new(*W.plane(-0.03, 40.0))
    state = None
    out = []
    for whole in (True, False):
        m = fgb.SpringyMesh.new(pos, idx, 0.01 * len(pos), 5.0, 0.01)
        if not faces:
            m.add_struts(np.stack([v[:, :-1].reshape(-1), v[:, 1:].reshape(-1)], 1)[::2], 4.0, 0.02)
        m.add_pins([0])
        m.set_precision(64)
        sim = fgb.Simulation.new([m], [obstacle])
        sim.set_config(cfg)
        sim.step(0)
        if state is None:
            state = m.get_points()
            state[:, 4:7] = rng.normal(0, 1.0, (len(pos), 3))
            state[:, 7:10] = rng.normal(0, 0.01, (len(pos), 3))
        m.set_points(state)
        for _ in range(4):
            if whole:
                sim.step(1)
            else:
                m.accumulate_forces(cfg)
                m.integrate(integration, 1.0 / 2000.0)
                m.update_points([obstacle], cfg)
                m.clear_forces()
        out.append(m.get_points_f64())
    assert np.isfinite(out[0]).all() and out[0].tobytes() == out[1].tobytes()
