"""The quick box and triangle tests in front of the reference's arithmetic
(pair_boxes, tri_surely_missed) against the oracle: rays aimed at the edges
and corners of triangles from sizes below the quick test's range to above
it, axis-parallel rays (which take the general box test), directions that
are not normalised and negative t_min (which take the general triangle
test). Hits, distances and occlusion flags are equal bit for bit."""
import numpy as np
import pytest

import oracle
from tracer_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(rng, n, size):
    sc = scenes.traversal(n, seed=int(rng.integers(1 << 30)))
    c = rng.uniform(-1, 1, (n, 1, 3)) * size * 4
    sc.positions = (c + rng.uniform(-1, 1, (n, 3, 3)) * size).astype(np.float32).reshape(-1, 3) + np.float32(0)
    flat = 3 * np.arange(n // 4)  # a quarter of them axis-aligned: boxes without thickness
    sc.positions[flat + 1, 0] = sc.positions[flat, 0]
    sc.positions[flat + 2, 0] = sc.positions[flat, 0]
    return sc


def _rays(rng, sc, n, size):
    """Aimed at points whose barycentric coordinates lie on an edge or a
    corner, within an ulp or so of one, or anywhere."""
    v = sc.positions.reshape(-1, 3, 3).astype(np.float64)[rng.integers(0, len(sc.positions) // 3, n)]
    b = rng.dirichlet(np.ones(3), n)
    kind = rng.integers(0, 5, n)
    b[kind == 0, 0] = 0.0
    b[kind == 1] = np.eye(3)[rng.integers(0, 3, (kind == 1).sum())]
    b[kind == 2, 1] = rng.choice([-1e-7, 1e-7, 3e-7], (kind == 2).sum())
    b /= b.sum(1, keepdims=True)
    at = (b[:, :, None] * v).sum(1)
    o = (at + rng.normal(size=(n, 3)) * size * rng.choice([1e-3, 1.0, 30.0], (n, 1))).astype(np.float32)
    d = at - o
    ax = kind == 4  # along an axis: reciprocals are infinite
    d[ax] = np.eye(3)[rng.integers(0, 3, ax.sum())] * rng.choice([-1.0, 1.0], (ax.sum(), 1))
    return scenes.make_rays(o, d / np.linalg.norm(d, axis=1, keepdims=True), 0.0, scenes.F32_MAX)


@pytest.mark.parametrize("size", [2.0 ** -24, 2.0 ** -19, 1.0, 1000.0, 2.0 ** 19, 2.0 ** 22])
@pytest.mark.parametrize("stretch,t_min", [(1.0, 0.0), (0.3, 0.0), (5.0, 1e-3), (1.0, -2.0)])
def test_hits_equal_the_oracle(gpu, size, stretch, t_min):
    rng = np.random.default_rng(int(np.log2(size) * 7) % 1000 + int(stretch * 10))
    sc = _scene(rng, 300, size)
    orc = oracle.Oracle(sc, "port")
    gpu.upload(sc)
    rays = _rays(rng, sc, 20000, size)
    rays["d"] *= np.float32(stretch)
    rays["t_min"] = np.float32(t_min * size)
    p0, t0 = orc.trace_closest(rays)
    p1, t1 = gpu.trace_closest(rays)
    assert (p0 >= 0).mean() > 0.2
    assert np.array_equal(p0, p1) and np.array_equal(t0.view(np.uint32), t1.view(np.uint32))
    for f in (0.5, 1.0, np.float32(1.0000001)):  # short, exactly at the hit, one ulp past it
        s = rays.copy()
        s["t_max"] = np.where(p0 >= 0, t0 * np.float32(f), np.float32(size * 3))
        assert np.array_equal(orc.trace_any(s), gpu.trace_any(s))
