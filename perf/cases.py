"""Performance cases: the work that programs built on this library have it do, through its public calls.

A case is one kind of call (or the few calls that a program always makes together) on one input. The
kinds and their sizes are those of the benchmark workloads, the benchmark harness stages and the tests:

  taylor     winding numbers of a query batch by the Taylor traversal (orders 0-2, plain and
             compensated near field; dense batches near the surface, sparse ones, a handful of queries)
  gradient   query gradient of the Taylor winding number
  exact      brute-force winding numbers
  adjoint    forward and backward pass: dL/dV and dL/dq of a loss over winding numbers
  frames     many moving meshes: refit, moment refit and queries of all of them, per frame
  build      BVH and moments of a mesh that has been uploaded
  distance   unsigned point-to-mesh distances
  ray        nearest ray hits
  antipodal  winding numbers and gradients by the antipodal method on an open mesh

Meshes are displaced UV spheres (closed) and "soups" made of them (a fifth of the triangles deleted,
a twentieth flipped), as in smallgwn_b200/meshes.py; queries are drawn on the GPU from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from smallgwn_b200 import api, meshes

INF = float("inf")


# ---- the cases --------------------------------------------------------------------------------------

def listed() -> list[dict]:
    return [
        # The benchmark's headline: a 1M-triangle mesh, 10M queries of which half lie at the surface,
        # compensated near field, accuracy for a maximum error of 1e-3. Offline voxelisation, remeshing.
        dict(name="taylor_dense", kind="taylor", mesh="sphere", phi=1024, theta=512, order=2, beta=3.5,
             compensated=True, mix="surface", n=10_000_000),
        # An ordinary batch with the default options and the harness's query mix (most of them far).
        dict(name="taylor_default", kind="taylor", mesh="sphere", phi=1024, theta=512, order=1, beta=2.0,
             compensated=False, mix="harness", n=1_000_003),
        # An interactive probe: a thousand points against a small mesh. Launches and latency.
        dict(name="taylor_few", kind="taylor", mesh="sphere", phi=64, theta=41, order=2, beta=2.0,
             compensated=False, mix="surface", n=1_000),
        # Normals and projection onto a level set of a triangle soup.
        dict(name="gradient_soup", kind="gradient", mesh="soup", phi=316, theta=316, order=2, beta=2.0,
             mix="surface", n=300_007),
        # The small exact workload: 5,120 triangles, 100,000 queries in a box around them.
        dict(name="exact_small", kind="exact", mesh="sphere", phi=64, theta=41, mix="box", n=100_000),
        # The differentiation workload: one optimisation step over a soup.
        dict(name="adjoint_soup", kind="adjoint", mesh="soup", phi=316, theta=316, order=1, beta=2.0, mix="surface",
             n=1_000_000),
        # One frame of a scene of moving meshes of uneven size (the batched workload, fewer meshes).
        dict(name="frames_scene", kind="frames", mesh="sphere", phi=160, theta=141, meshes=24, order=1, beta=2.0,
             mix="surface", n=2_000_003),
        # Loading a large mesh: H-PLOC tree and order-2 moments.
        dict(name="build_large", kind="build", mesh="sphere", phi=1024, theta=512, method="hploc", order=2),
        # Loading a small one: LBVH tree and order-1 moments. Launches and latency.
        dict(name="build_small", kind="build", mesh="sphere", phi=64, theta=41, method="lbvh", order=1),
        # Signed-distance grids and collision checks: distances of an ordered batch.
        dict(name="distance_sorted", kind="distance", mesh="sphere", phi=1024, theta=512, mix="surface",
             band=INF, ordered=True, n=2_000_000),
        # Visibility and picking: incoherent rays from the neighbourhood of the mesh.
        dict(name="ray_mixed", kind="ray", mesh="sphere", phi=1024, theta=512, mix="surface", n=4_000_001),
        # The antipodal workload on an open mesh with thousands of boundary edges: value and gradient.
        dict(name="antipodal_open", kind="antipodal", mesh="soup", phi=80, theta=80, mix="surface", n=200_000),
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """Another case of the listed kinds, over the sizes and options that they stand for."""
    kind = rng.choice(["taylor", "taylor", "taylor", "gradient", "exact", "adjoint", "frames", "build", "build",
                       "distance", "ray", "antipodal"])
    c = dict(kind=kind)
    if kind in ("taylor", "distance", "ray", "build"):
        c["mesh"] = rng.choice(["sphere", "sphere", "soup"])
        c["phi"] = _log_uniform(rng, 24, 1024)
        c["theta"] = max(9, min(512, c["phi"] // rng.choice([1, 2, 3])))
    if kind == "taylor":
        c.update(order=rng.choice([0, 1, 2]), beta=rng.choice([1.5, 2.0, 3.0, 3.5]), compensated=rng.random() < 0.4,
                 mix=rng.choice(["surface", "harness", "box"]), n=_log_uniform(rng, 200, 6_000_000))
    elif kind == "gradient":
        p = _log_uniform(rng, 24, 400)
        c.update(mesh=rng.choice(["sphere", "soup"]), phi=p, theta=p, order=rng.choice([0, 1, 2]), beta=2.0,
                 mix=rng.choice(["surface", "box"]), n=_log_uniform(rng, 1_000, 1_000_000))
    elif kind == "exact":
        p = _log_uniform(rng, 12, 90)
        n = _log_uniform(rng, 100, 300_000)
        c.update(mesh=rng.choice(["sphere", "soup"]), phi=p, theta=p, mix=rng.choice(["box", "surface"]),
                 n=max(1, min(n, 2_000_000_000 // (2 * p * p))))
    elif kind == "adjoint":
        p = _log_uniform(rng, 24, 316)
        c.update(mesh=rng.choice(["sphere", "soup"]), phi=p, theta=p, order=rng.choice([0, 1]), beta=2.0,
                 mix=rng.choice(["surface", "box"]), n=_log_uniform(rng, 1_000, 1_000_000))
    elif kind == "frames":
        p = _log_uniform(rng, 24, 160)
        c.update(mesh="sphere", phi=p, theta=max(9, p - 11), meshes=rng.randint(2, 24), order=rng.choice([0, 1, 2]),
                 beta=2.0, mix=rng.choice(["surface", "box"]), n=_log_uniform(rng, 10_000, 2_000_000))
    elif kind == "build":
        c.update(method=rng.choice(["hploc", "lbvh"]), order=rng.choice([0, 1, 2]))
    elif kind == "distance":
        c.update(mix=rng.choice(["surface", "box"]), band=rng.choice([INF, INF, 0.05]), ordered=rng.random() < 0.7,
                 n=_log_uniform(rng, 1_000, 2_000_000))
    elif kind == "ray":
        c.update(mix=rng.choice(["surface", "box"]), n=_log_uniform(rng, 1_000, 4_000_000))
    elif kind == "antipodal":
        p = _log_uniform(rng, 24, 80)
        c.update(mesh="soup", phi=p, theta=p, mix=rng.choice(["surface", "box"]), n=_log_uniform(rng, 1_000, 200_000))
    return c


# ---- inputs -----------------------------------------------------------------------------------------

def _mesh(kind: str, phi: int, theta: int, seed: int) -> dict:
    """SoA arrays (float32 x, y, z; uint32 i0, i1, i2) on the host, as a loader would hand them over."""
    V, F = meshes.uv_sphere(phi, theta, seed)
    if kind == "soup":
        rng = np.random.default_rng(seed)
        F = F[rng.uniform(size=F.shape[0]) >= 0.2]
        flip = rng.uniform(size=F.shape[0]) < 0.05
        F[flip] = F[flip][:, [0, 2, 1]]
    return meshes.to_soa(V, F)


def _rescaled(m: dict, seed: int) -> dict:
    """The mesh at another scale (a power of two) with its vertices numbered from another one on: new
    arrays, and a tree of the same size."""
    rng = np.random.default_rng(seed)
    scale, shift = np.float32(2.0 ** int(rng.integers(-12, 13))), int(rng.integers(0, m["x"].size))
    out = {k: np.roll(m[k], shift) * scale for k in "xyz"}
    out.update({k: ((m[k].astype(np.int64) + shift) % m["x"].size).astype(np.uint32) for k in ("i0", "i1", "i2")})
    return out


def _mesh_tensors(m: dict) -> tuple[torch.Tensor, torch.Tensor]:
    V = torch.from_numpy(np.stack([m["x"], m["y"], m["z"]], axis=1)).cuda()
    F = torch.from_numpy(np.stack([m["i0"], m["i1"], m["i2"]], axis=1).astype(np.int64)).cuda()
    return V, F


def _points(V: torch.Tensor, F: torch.Tensor, mix: str, n: int, gen: torch.Generator) -> list[torch.Tensor]:
    """Query points of a mix, shuffled, as three contiguous tensors.

    surface: half uniform in the bounding box scaled by 1.2, half at a surface sample offset along the
             triangle's normal by N(0, 1e-3);
    harness: 70 % centre + U(-0.85, 0.85) extents, 30 % centre + (+-U(1.5, 3) + U(-0.25, 0.25)) extents;
    box:     uniform in the bounding box scaled by 1.5.
    """
    lo, hi = V.amin(0), V.amax(0)
    mid, ext = (lo + hi) * 0.5, hi - lo

    def uni(k, a, b):
        return a + (b - a) * torch.rand(k, 3, generator=gen, device="cuda")

    if mix == "box":
        q = mid + uni(n, -0.75, 0.75) * ext
    elif mix == "harness":
        far = n * 3 // 10
        sign = torch.where(uni(far, 0.0, 1.0) < 0.5, -1.0, 1.0)
        q = torch.cat([mid + uni(n - far, -0.85, 0.85) * ext,
                       mid + (sign * uni(far, 1.5, 3.0) + uni(far, -0.25, 0.25)) * ext])
    else:
        box = n // 2
        srf = n - box
        t = F[torch.randint(0, F.shape[0], (srf,), generator=gen, device="cuda")]
        a, b, c = V[t[:, 0]], V[t[:, 1]], V[t[:, 2]]
        u = torch.rand(srf, 2, generator=gen, device="cuda")
        u = torch.where(u.sum(1, keepdim=True) > 1.0, 1.0 - u, u)
        nrm = torch.linalg.cross((b - a).double(), (c - a).double())
        nrm = nrm / nrm.norm(dim=1, keepdim=True).clamp_min(1e-30)
        off = 1e-3 * torch.randn(srf, 1, generator=gen, device="cuda")
        q = torch.cat([mid + uni(box, -0.6, 0.6) * ext,
                       a + u[:, :1] * (b - a) + u[:, 1:] * (c - a) + off * nrm.float()])
    q = q[torch.randperm(n, generator=gen, device="cuda")]
    return [q[:, k].contiguous() for k in range(3)]


def _directions(n: int, gen: torch.Generator) -> list[torch.Tensor]:
    d = torch.randn(n, 3, generator=gen, device="cuda")
    d = d / d.norm(dim=1, keepdim=True).clamp_min(1e-12)
    return [d[:, k].contiguous() for k in range(3)]


def _ok(status: api.gwn_status) -> None:
    if not status.is_ok():
        raise RuntimeError(status.message)


class _device_array:
    """A device array of a library object as the CUDA array interface describes it; keeps the object."""

    def __init__(self, owner, ptr: int, shape: tuple, typestr: str) -> None:
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(int(ptr), False), version=3)


def _view(owner, ptr: int, shape: tuple, typestr: str) -> torch.Tensor:
    return torch.as_tensor(_device_array(owner, ptr, shape, typestr), device="cuda")


def _moment_view(m: api.gwn_bvh4_moment_object) -> torch.Tensor:
    v = m.accessor()
    return _view(m, v.nodes, (int(v.node_count), {0: 7, 1: 13, 2: 23}[m.order], 4), "<f4")


def _node_view(b: api.gwn_bvh4_object) -> torch.Tensor:
    v = b.accessor()
    return _view(b, v.nodes, (int(v.node_count), 4, 8), "<i4")  # six bounds and a 64-bit reference per child


def _upload(m: dict) -> api.gwn_geometry_object:
    g = api.gwn_geometry_object()
    _ok(api.gwn_upload_geometry(g, m["x"], m["y"], m["z"], m["i0"], m["i1"], m["i2"]))
    return g


def _method(name: str) -> api.gwn_bvh_build_options:
    k = api.gwn_bvh_build_method.k_lbvh if name == "lbvh" else api.gwn_bvh_build_method.k_hploc
    return api.gwn_bvh_build_options(method=k)


def _tree(g, order: int | None) -> tuple:
    b = api.gwn_bvh4_object()
    _ok(api.gwn_build_bvh(g, b))
    if order is None:
        return b, None
    m = api.gwn_bvh4_moment_object(order)
    _ok(api.gwn_refit_bvh_moment(order, b, m))
    return b, m


def _frames_state(case: dict, seed: int, gen: torch.Generator) -> dict:
    """Meshes of uneven size in one shared vertex buffer; the frame's positions beside it. The rest
    shapes, from which the trees are built, are the same for every seed."""
    hosts = []
    for i in range(case["meshes"]):
        phi = max(12, case["phi"] * (4 + i % 5) // 8)
        theta = max(8, case["theta"] * (4 + i % 3) // 6)
        hosts.append(_mesh(case["mesh"], phi, theta, 100 + i))
    per = case["n"] // case["meshes"]
    counts = [per] * (case["meshes"] - 1) + [case["n"] - per * (case["meshes"] - 1)]
    rest = torch.from_numpy(np.stack([np.concatenate([h[k] for h in hosts]) for k in "xyz"])).cuda()
    # the frame's pose: a smooth swelling of up to 2 % of the radius
    pose = rest * (1.0 + 0.02 * torch.sin(5.0 * rest[2] + 3.0 * rest[0] + float(seed % 1009)))
    live = rest.clone()
    winding = torch.empty(case["n"], device="cuda")
    entries, nodes, moments, at, first = [], [], [], 0, 0
    for h, count in zip(hosts, counts):
        V, F = _mesh_tensors(h)
        q = _points(V, F, case["mix"], count, gen)
        idx = [F[:, k].to(torch.int32).contiguous() for k in range(3)]
        x, y, z = (live[k, at:at + h["x"].size] for k in range(3))
        g = api.gwn_geometry_view(x, y, z, *idx)
        b, m = _tree(g, case["order"])
        entries.append((g, b, m, *q, winding[first:first + count]))
        nodes.append(_node_view(b))
        moments.append(_moment_view(m))
        at += h["x"].size
        first += count
    batch = api.gwn_batch(entries, accuracy_scale=case["beta"])
    _ok(batch.status)
    return dict(live=live, pose=pose, batch=batch, outputs=dict(winding=winding, nodes=nodes, moments=moments))


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 7919 + 17)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "frames":
        s.update(_frames_state(case, seed, gen))
        return s
    if kind == "build":  # one shape at other scales, so that the arrays of the tree have the same size
        s["geometry"] = _upload(_rescaled(_mesh(case["mesh"], case["phi"], case["theta"], 2), seed))
        s["options"] = _method(case["method"])
        return s
    host = _mesh(case["mesh"], case["phi"], case["theta"], seed)
    s["geometry"] = g = _upload(host)
    V, F = _mesh_tensors(host)
    n = case["n"]
    s["q"] = _points(V, F, case["mix"], n, gen)
    s["bvh"], s["moment"] = _tree(g, case.get("order"))
    if kind == "gradient":
        s["out"] = [torch.empty(n, device="cuda") for _ in range(3)]
    elif kind == "ray":
        s["d"] = _directions(n, gen)
        s["out"] = torch.empty(n, 8, device="cuda")
    elif kind == "adjoint":
        s["out"] = torch.empty(n, device="cuda")
        s["grad"] = torch.randn(n, generator=gen, device="cuda")
        s["dv"] = [torch.empty(V.shape[0], device="cuda") for _ in range(3)]
        s["dq"] = [torch.empty(n, device="cuda") for _ in range(3)]
    elif kind == "antipodal":
        s["chain"] = api.gwn_boundary_chain_object()
        _ok(api.gwn_build_boundary_chain(g, s["chain"]))
        s["out"] = torch.empty(n, device="cuda")
        s["gradient"] = [torch.empty(n, device="cuda") for _ in range(3)]
    else:
        s["out"] = torch.empty(n, device="cuda")
    return s


# ---- one pass ---------------------------------------------------------------------------------------

def run(state: dict):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "taylor":
        near = api.near_precision.compensated if c["compensated"] else api.near_precision.plain
        _ok(api.gwn_compute_winding_number_taylor_batch(c["order"], s["bvh"], s["moment"], *s["q"], s["out"],
                                                        accuracy_scale=c["beta"], precision=near))
        return s["out"]
    if kind == "gradient":
        _ok(api.gwn_compute_winding_gradient_taylor_batch(c["order"], s["bvh"], s["moment"], *s["q"], *s["out"],
                                                          accuracy_scale=c["beta"]))
        return s["out"]
    if kind == "exact":
        _ok(api.gwn_compute_winding_number_exact_batch(s["bvh"], *s["q"], s["out"]))
        return s["out"]
    if kind == "adjoint":
        st, saved = api.gwn_winding_taylor_forward(c["order"], s["bvh"], s["moment"], *s["q"], s["out"],
                                                   accuracy_scale=c["beta"])
        _ok(st)
        _ok(api.gwn_winding_taylor_backward(saved, s["geometry"], s["bvh"], s["moment"], s["grad"], *s["dv"],
                                            *s["dq"]))
        return dict(winding=s["out"], dv=s["dv"], dq=s["dq"])
    if kind == "frames":
        s["live"].copy_(s["pose"])
        _ok(s["batch"].frame())
        return s["outputs"]
    if kind == "build":
        b = api.gwn_bvh4_object()
        _ok(api.gwn_build_bvh(s["geometry"], b, s["options"]))
        m = api.gwn_bvh4_moment_object(c["order"])
        _ok(api.gwn_refit_bvh_moment(c["order"], b, m))
        v = b.accessor()
        return dict(nodes=_node_view(b), order=_view(b, v.primitive_indices, (int(v.primitive_count),), "<i4"),
                    triangles=_view(b, v.triangles, (int(v.primitive_count), 9), "<f4"), moments=_moment_view(m))
    if kind == "distance":
        _ok(api.gwn_compute_unsigned_distance_batch(s["bvh"], *s["q"], s["out"], culling_band=c["band"],
                                                    sort_queries=c["ordered"]))
        return s["out"]
    if kind == "ray":
        _ok(api.gwn_compute_ray_first_hit_batch(s["bvh"], *s["q"], *s["d"], s["out"]))
        words = s["out"].view(torch.int32)
        return dict(hit=s["out"][:, :6], triangle=words[:, 6], status=words[:, 7])
    if kind == "antipodal":
        _ok(api.gwn_compute_winding_number_antipodal_batch(s["geometry"], s["bvh"], s["chain"], *s["q"], s["out"]))
        _ok(api.gwn_compute_winding_gradient_antipodal_batch(s["geometry"], s["chain"], *s["q"], *s["gradient"]))
        return dict(winding=s["out"], gradient=s["gradient"])
    raise ValueError(kind)


# ---- what a pass cannot do without -------------------------------------------------------------------

_MOMENT_BYTES = {0: 112, 1: 208, 2: 368}  # per node, the published layout


def _triangles(case: dict) -> float:
    t = 2.0 * case["phi"] * (case["theta"] - 1)
    return 0.8 * t if case["mesh"] == "soup" else t


def work(case: dict) -> dict:
    """Bytes: every input read and every output written once. Operations: for the traversals an
    estimate of the far-field terms, exact triangles, box and triangle tests of a query (from the
    traversal statistics: about 48 far-field terms per unit of the squared accuracy scale at a million
    triangles, growing with the logarithm of the size); for the brute-force paths their pairs."""
    kind = case["kind"]
    t = _triangles(case)
    n = float(case.get("n", 0))
    nodes = 0.5 * t
    depth = math.log2(max(t, 16.0)) / 20.0
    if kind == "frames":
        t *= case["meshes"] * 0.6
        nodes = 0.5 * t
    tree = 128.0 * nodes + 36.0 * t
    order = case.get("order", 0)
    if order is None:
        order = 0
    far = 48.0 * depth * case.get("beta", 2.0) ** 2
    terms = far * {0: 21.0, 1: 36.0, 2: 62.0}[order] + 45.0 * 60.0
    if kind == "taylor":
        return dict(bytes=16.0 * n + 36.0 * t + _MOMENT_BYTES[order] * nodes, flops=n * terms)
    if kind == "gradient":
        return dict(bytes=24.0 * n + 36.0 * t + _MOMENT_BYTES[order] * nodes, flops=2.0 * n * terms)
    if kind == "exact":
        return dict(bytes=16.0 * n + 36.0 * t, flops=70.0 * n * t)
    if kind == "adjoint":
        return dict(bytes=44.0 * n + 2.0 * (36.0 * t + _MOMENT_BYTES[order] * nodes) + 12.0 * 0.5 * t,
                    flops=4.0 * n * terms)
    if kind == "frames":
        return dict(bytes=16.0 * n + 24.0 * 0.5 * t + 12.0 * t + 2.0 * tree + _MOMENT_BYTES[order] * nodes,
                    flops=n * terms + 400.0 * t)
    if kind == "build":
        return dict(bytes=12.0 * 0.5 * t + 12.0 * t + tree + 4.0 * t + _MOMENT_BYTES[order] * nodes, flops=600.0 * t)
    if kind == "distance":
        return dict(bytes=16.0 * n + tree, flops=n * 60.0 * 4.0 * 20.0 * depth)
    if kind == "ray":
        return dict(bytes=56.0 * n + tree, flops=n * 18.0 * 4.0 * 24.0 * depth)
    if kind == "antipodal":
        rows = 0.7 * t if case["mesh"] == "soup" else 2.0 * case["phi"]
        return dict(bytes=28.0 * n + 16.0 * rows + tree, flops=n * rows * (40.0 + 90.0))
    raise ValueError(kind)


# ---- how far two right answers may lie apart ----------------------------------------------------------

def tolerance(case: dict):
    """32-bit arithmetic throughout, about four times what reruns, the other near-field form or the
    64-bit answer showed."""
    kind = case["kind"]
    if kind == "ray":
        # one fixed operation order per triangle; among equally near hits the lower id
        return dict(rel=1e-5, differ=1e-5)
    if kind == "distance":
        return dict(rel=1e-6)
    if kind == "exact":
        # sums in 64 bits, cancelling pairs in 64 bits: 2e-8 to 1.3e-7 from the 64-bit answer
        return dict(rel=1e-6)
    if kind == "adjoint" and case["mesh"] == "sphere":
        # closed meshes end in degenerate triangles at the poles, whose terms cancel: the atomic sums of
        # two runs of one program differ by up to 7e-5
        return dict(rel=3e-4)
    if kind in ("taylor", "frames", "gradient") and case["mix"] == "surface" and not case.get("compensated", False):
        # the plain near field loses digits where a query lies close to a triangle that is large beside
        # its distance: up to 3.4e-4 between the plain and the compensated form on coarse meshes
        return dict(rel=1e-3)
    # sums of hundreds to thousands of 32-bit terms: 2e-7 to 2.4e-6. The trees of the builds are whole
    # numbers and exact; their moments are such sums.
    return dict(rel=1e-5)


# ---- 64-bit answers ----------------------------------------------------------------------------------

def _chunks(n: int, m: int, budget: int = 60_000_000):
    step = max(1, budget // max(m, 1))
    for i in range(0, n, step):
        yield slice(i, min(n, i + step))


def _winding64(V: torch.Tensor, F: torch.Tensor, q: torch.Tensor) -> torch.Tensor:
    """Sum of the solid angles of all triangles over 4 pi."""
    A, B, C = V[F[:, 0]], V[F[:, 1]], V[F[:, 2]]
    out = torch.empty(q.shape[0], dtype=torch.float64, device=q.device)
    for sl in _chunks(q.shape[0], F.shape[0]):
        p = q[sl, None, :]
        ax, ay, az = (A[None, :, k] - p[..., k] for k in range(3))
        bx, by, bz = (B[None, :, k] - p[..., k] for k in range(3))
        cx, cy, cz = (C[None, :, k] - p[..., k] for k in range(3))
        la = (ax * ax + ay * ay + az * az).sqrt()
        lb = (bx * bx + by * by + bz * bz).sqrt()
        lc = (cx * cx + cy * cy + cz * cz).sqrt()
        num = ax * (by * cz - bz * cy) + ay * (bz * cx - bx * cz) + az * (bx * cy - by * cx)
        den = la * lb * lc
        den += (ax * bx + ay * by + az * bz) * lc
        den += (ax * cx + ay * cy + az * cz) * lb
        den += (bx * cx + by * cy + bz * cz) * la
        ang = torch.atan2(num, den)
        ang[(num == 0) | (la == 0) | (lb == 0) | (lc == 0)] = 0.0
        out[sl] = ang.sum(1) * (2.0 / (4.0 * math.pi))
    return out


def _boundary(F: np.ndarray) -> tuple[np.ndarray, np.ndarray, np.ndarray]:
    """Directed edges of the mesh whose two directions do not cancel: (start, end, multiplicity)."""
    e = np.concatenate([F[:, [0, 1]], F[:, [1, 2]], F[:, [2, 0]]]).astype(np.int64)
    lo, hi = e.min(1), e.max(1)
    key = lo << 32 | hi
    uniq, inv = np.unique(key, return_inverse=True)
    net = np.bincount(inv, weights=np.sign(e[:, 1] - e[:, 0]), minlength=uniq.size)
    keep = net != 0
    a, b, m = uniq[keep] >> 32, uniq[keep] & 0xFFFFFFFF, net[keep]
    return np.where(m > 0, a, b), np.where(m > 0, b, a), np.abs(m)


def _boundary_gradient64(V: torch.Tensor, F: torch.Tensor, q: torch.Tensor) -> list[torch.Tensor]:
    """Gradient of the winding number: the line integral of (x - q) x dx / |x - q|^3 along the boundary."""
    a, b, m = (torch.from_numpy(x).to(V.device) for x in _boundary(F.cpu().numpy()))
    out = [torch.zeros(q.shape[0], dtype=torch.float64, device=q.device) for _ in range(3)]
    if a.numel() == 0:
        return out
    S, E = V[a], V[b]
    for sl in _chunks(q.shape[0], a.numel()):
        p = q[sl, None, :]
        sx, sy, sz = (S[None, :, k] - p[..., k] for k in range(3))
        ex, ey, ez = (E[None, :, k] - p[..., k] for k in range(3))
        ls = (sx * sx + sy * sy + sz * sz).sqrt()
        le = (ex * ex + ey * ey + ez * ez).sqrt()
        # |s||e| + s.e without cancellation where the edge passes the query: |s x e|^2 / (|s||e| - s.e)
        cr = (sy * ez - sz * ey, sz * ex - sx * ez, sx * ey - sy * ex)
        dt = sx * ex + sy * ey + sz * ez
        pr = ls * le
        c2 = cr[0] ** 2 + cr[1] ** 2 + cr[2] ** 2
        f = torch.where(dt >= 0, 1.0 / (pr + dt), (pr - dt) / c2) * (ls + le) / pr * m
        for k in range(3):
            out[k][sl] = (f * cr[k]).sum(1) / (4.0 * math.pi)
    return out


def exact(case: dict, seed: int):
    """What run() returns, in 64 bits, for the brute-force paths. The Taylor paths' 64-bit answer would
    need a traversal of the same tree with the same decisions, and the distances and hits a search
    over all pairs: None."""
    kind = case["kind"]
    if kind not in ("exact", "antipodal"):
        return None
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 7919 + 17)
    V, F = _mesh_tensors(_mesh(case["mesh"], case["phi"], case["theta"], seed))
    q = torch.stack(_points(V, F, case["mix"], case["n"], gen), dim=1).double()
    w = _winding64(V.double(), F, q)
    if kind == "exact":
        return w
    return dict(winding=w, gradient=_boundary_gradient64(V.double(), F, q))
