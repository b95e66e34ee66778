"""The exact batch takes its triangles two at a time: sizes around the edges of pairs, tiles and blocks, and queries that leave the
packed path (on vertices, in a triangle's plane, on an edge, on an edge's line, far away)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from smallgwn_b200 import meshes
from test_gpu_build import build, upload
from test_gpu_query import run_exact

pytestmark = pytest.mark.gpu

# The packed and the general form evaluate the same float records; the error against FP64 is that of the
# records' float edges (below 5e-6 on meshes of this size, as for the other exact batches).
EXACT_TOL = 5e-6


def part(triangles: int) -> dict:
    """The first triangles of a small displaced sphere: open, of any size."""
    V, F = meshes.uv_sphere(24, 24, 5)
    assert triangles <= F.shape[0]
    return meshes.to_soa(V, F[:triangles])


def probes(mesh: dict, n: int, seed: int) -> np.ndarray:
    """Queries around the mesh, some of them on vertices, edge midpoints, triangle centroids (in the
    triangle's plane up to rounding), on an edge's extension, and far away."""
    rng = np.random.default_rng(seed)
    P = np.stack([mesh[k] for k in "xyz"], 1).astype(np.float64)
    T = np.stack([mesh[k] for k in ("i0", "i1", "i2")], 1)[rng.integers(0, mesh["i0"].size, n)]
    a, b, c = P[T[:, 0]], P[T[:, 1]], P[T[:, 2]]
    kinds = np.stack([a + rng.uniform(-0.3, 0.3, (n, 3)), a, (a + b) / 2, (a + b + c) / 3, b + 1.5 * (b - a),
                      rng.uniform(-50, 50, (n, 3)), a + rng.uniform(-0.3, 0.3, (n, 3)) * 1e-2,
                      rng.uniform(-1.5, 1.5, (n, 3))])
    return np.ascontiguousarray(kinds[rng.integers(0, 8, n), np.arange(n)].T.astype(np.float32))


@pytest.mark.parametrize("triangles", [1, 2, 3, 255, 256, 257, 511, 513, 1000])
@pytest.mark.parametrize("n", [1, 511, 1025])
def test_exact_batch_sizes(cuda, triangles, n):
    mesh = part(triangles)
    bvh = build(upload(mesh))
    q = probes(mesh, n, seed=triangles + n)
    got = run_exact(cuda, bvh, q)
    want = oracle.exact_winding(mesh, *q.astype(np.float64), fp64=True)
    # on the surface itself the winding number jumps: a query there up to its coordinates' rounding has
    # the value of either side
    off = oracle.mesh_distance(mesh, *q) >= 1e-6
    assert np.isfinite(got).all()
    assert (np.abs(got - want) <= EXACT_TOL)[off].all()


@pytest.mark.parametrize("scale", [1e-12, 1e12])
def test_exact_batch_scales(cuda, scale):
    """Products of three lengths near the ends of the float range: the arguments are formed from
    normalised directions, as good as at scale 1."""
    mesh = part(301)
    q = probes(mesh, 700, seed=9)
    want = oracle.exact_winding(mesh, *q.astype(np.float64), fp64=True)
    far = oracle.mesh_distance(mesh, *q) > 0.05
    scaled = dict(mesh, **{k: (mesh[k] * np.float32(scale)).astype(np.float32) for k in "xyz"})
    got = run_exact(cuda, build(upload(scaled)), (q * np.float32(scale)).astype(np.float32))
    assert (np.abs(got - want) <= EXACT_TOL)[far].all()
