"""Performance cases: the calls that programs make of this engine, over the sizes they make them at.

A case is a dict of plain values; ``kind`` names the entry point it goes through:

  dense    ``extract_tensor`` on a CUDA grid (quads, or triangles with ``triangles``)
  host     ``extract``: host grid in, host mesh out
  batch    ``extract_batch``: many grids of uneven sizes in one call
  fit      ``dual_contour`` forward and backward: one step of fitting a grid to a surface
  refine   ``extract_tensor`` with ContouringMethod.Ours
  sparse   ``extract_tensor`` of the brick backend (``multi``: up to two vertices per cell)
  mesh     ``mesh_to_sdf_tensor`` (``voxelize``: signs from a voxel solid)
  post     ``postprocess_mesh_tensor``: weld, largest component, hole filling

A program keeps one backend and hands it grid after grid, so the states of one case share a
backend (one per case, made on its first ``prepare``).
"""
import json
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "phanty-sdf-cuda_b200"))

from contouring_b200 import (B200DualContouringBackend, B200SparseDualContouringBackend,  # noqa: E402
                             ContouringMethod, ContouringOptions, DenseSdfGrid, NormalComputationMode,
                             dual_contour, mesh_to_sdf_tensor, postprocess_mesh_tensor, synth)

BATCH_SIZES = (32, 48, 64, 96, 128, 192)        # the resolutions of the 256-grid benchmark


def listed():
    return [
        # a preview of a small object: the smallest call, all launches and latency
        {"name": "dense 32", "kind": "dense", "scene": 0, "nx": 32, "ny": 32, "nz": 32, "triangles": False},
        # a cropped scan: odd, uneven sizes, and the triangles most viewers want
        {"name": "dense 161x118x97 tri", "kind": "dense", "scene": 3, "nx": 161, "ny": 118, "nz": 97, "triangles": True},
        # the headline benchmark's grid
        {"name": "dense 1024", "kind": "dense", "scene": 0, "nx": 1024, "ny": 1024, "nz": 1024, "triangles": False},
        # the drop-in call on an ordinary grid: upload, extraction, download
        {"name": "host 256", "kind": "host", "scene": 1, "nx": 256, "ny": 256, "nz": 256},
        # a dataset's shapes at uneven resolutions, one call
        {"name": "batch 32 grids", "kind": "batch", "scene": 7, "count": 32},
        # one step of fitting a grid, the size of the adjoint benchmark
        {"name": "fit 128", "kind": "fit", "scene": 0, "res": 128},
        # the refinement of its benchmark's size with all its inner iterations
        {"name": "refine 128", "kind": "refine", "scene": 0, "res": 128, "outer": 20, "inner": 100},
        # the reference CLI's default GPU backend on a large grid
        {"name": "sparse 512", "kind": "sparse", "scene": 0, "nx": 512, "ny": 512, "nz": 512, "brick": 8, "mode": 0,
         "multi": False},
        # its multi-vertex variant on an odd grid with another brick size and normal mode
        {"name": "sparse 193x150x121 multi", "kind": "sparse", "scene": 2, "nx": 193, "ny": 150, "nz": 121, "brick": 5,
         "mode": 1, "multi": True},
        # the mesh conversion's benchmark: 163,840 triangles into 512^3 points
        {"name": "mesh 512", "kind": "mesh", "res": 512, "spheres": 32, "subdiv": 4, "voxelize": False},
        # the conversion of one object at a preview size, voxel signs
        {"name": "mesh 100 voxels", "kind": "mesh", "res": 100, "spheres": 8, "subdiv": 3, "voxelize": True},
        # clean-up of an extracted mesh before export
        {"name": "post 512", "kind": "post", "scene": 0, "nx": 512, "ny": 512, "nz": 512, "holes": True,
         "floaters": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    """Three sizes within a factor of two of one another, log-uniform, odd ones among them."""
    top = _log(rng, lo, hi)
    return dict(zip(("nx", "ny", "nz"), (max(lo, round(top * rng.uniform(0.5, 1.0))) for _ in range(3))))


def draw(rng):
    kind = rng.choice(("dense", "dense", "host", "batch", "fit", "refine", "sparse", "mesh", "post"))
    if kind == "mesh":
        return {"kind": kind, "res": _log(rng, 32, 400), "spheres": _log(rng, 1, 32), "subdiv": rng.randint(2, 4),
                "voxelize": rng.random() < 0.5}
    c = {"kind": kind, "scene": rng.randrange(1000)}
    if kind == "dense":
        return {**c, **_dims(rng, 16, 1000), "triangles": rng.random() < 0.3}
    if kind == "host":
        return {**c, **_dims(rng, 16, 400)}
    if kind == "batch":
        return {**c, "count": _log(rng, 2, 32)}
    if kind == "fit":
        return {**c, "res": _log(rng, 24, 256)}
    if kind == "refine":
        return {**c, "res": _log(rng, 64, 144), "outer": rng.randint(1, 4), "inner": rng.choice((20, 50, 100))}
    if kind == "sparse":
        return {**c, **_dims(rng, 16, 640), "brick": rng.choice((4, 5, 8, 16)), "mode": rng.randrange(3),
                "multi": rng.random() < 0.5}
    return {**c, **_dims(rng, 32, 640), "holes": rng.random() < 0.7, "floaters": rng.random() < 0.7}


# ---- inputs ------------------------------------------------------------------------------
# The case fixes the scene and with it how many vertices and quads come out; the seed changes
# the values.

def _csg(case):
    """The middle nx x ny x nz points of a sharp-feature CSG scene sampled at the largest of
    the three sizes on [-0.5, 0.5]^3."""
    dims = (case["nx"], case["ny"], case["nz"])
    res = max(dims)
    i0, j0, k0 = ((res - d) // 2 for d in dims)
    vals, _, sp, org = synth.csg(res, seed=case["scene"], device="cuda", planes=(k0, k0 + dims[2]))
    vals = vals.view(dims[2], res, res)[:, j0:j0 + dims[1], i0:i0 + dims[0]].contiguous().view(-1)
    org = tuple(float(np.float32(o + a * h)) for o, a, h in zip(org, (i0, j0, k0), sp))
    return vals, dims, sp, org


def _rbf(case):
    return synth.rbf_sphere(case["res"], seed=case["scene"], device="cuda")


def _varied(grid, seed, depth):
    """The grid's values times a smooth positive field of the seed's, 1 +- depth along each
    axis: every value keeps its sign, so the cells crossed are the scene's, the crossings move."""
    vals, dims, sp, org = grid
    rng = np.random.default_rng(seed)
    v = vals.view(dims[2], dims[1], dims[0])
    for axis, n in enumerate(v.shape):
        x = torch.linspace(0, 2 * math.pi * rng.uniform(2, 8), n) + rng.uniform(0, 2 * math.pi)
        v.mul_((1 + depth * x.sin()).cuda().view([n if d == axis else 1 for d in range(3)]))
    return vals, dims, sp, org


def _scaled(grid, seed):
    """The same scene in another unit, inside and outside exchanged for odd seeds. The sparse
    backends compare values with the spacing: a power of two leaves what they decide alone."""
    vals, dims, sp, org = grid
    unit = 2.0 ** (seed % 41 - 20)
    return vals.mul_(-unit if seed % 2 else unit), dims, tuple(h * unit for h in sp), tuple(o * unit for o in org)


def _batch_sizes(case):
    rng = np.random.default_rng(case["scene"])
    return [int(rng.choice(BATCH_SIZES)) for _ in range(case["count"])]


def _grids(case, seed):
    if case["kind"] == "batch":
        return [_varied(synth.csg(r, seed=1000 * case["scene"] + b, device="cuda"), 100 * seed + b, 0.2)
                for b, r in enumerate(_batch_sizes(case))]
    if case["kind"] == "sparse":
        return [_scaled(_csg(case), seed)]
    if case["kind"] == "refine":                                # spheres are read from the values: near distances
        return [_varied(_rbf(case), seed, 0.01)]
    return [_varied(_rbf(case) if case["kind"] == "fit" else _csg(case), seed, 0.2)]


_backends = {}


def _backend(case):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    if key not in _backends:
        if case["kind"] == "sparse":
            _backends[key] = B200SparseDualContouringBackend(case["brick"], NormalComputationMode(case["mode"]), 0,
                                                             case["multi"])
        else:
            o = ContouringOptions()
            o.emit_triangles = bool(case.get("triangles", False))
            if case["kind"] == "refine":
                o.method = ContouringMethod.Ours
                o.outer_iters, o.inner_iters = case["outer"], case["inner"]
            _backends[key] = B200DualContouringBackend(0, o)
    return _backends[key]


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "backend": _backend(case)}
    if kind in ("dense", "sparse", "refine"):
        s["grid"], = _grids(case, seed)
    elif kind == "host":
        (vals, dims, sp, org), = _grids(case, seed)
        s["grid"] = DenseSdfGrid(*dims, *sp, *org, values=vals.cpu().pin_memory().numpy())
    elif kind == "batch":
        s["grids"] = _grids(case, seed)
    elif kind == "fit":
        (vals, *s["where"]), = _grids(case, seed)
        s["values"] = vals.requires_grad_(True)
    elif kind == "mesh":
        V, F = synth.icosphere_scene(case["spheres"], case["subdiv"], seed)
        s["dims"], s["spacing"], s["origin"] = synth.mesh_grid(V, case["res"])
        s["vertices"], s["faces"] = torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda()
        s["voxelize"] = case["voxelize"]
    else:
        # welding and filling compare lengths: an extracted mesh in another unit per seed
        V, s["faces"], _ = s["backend"].extract_tensor(*_csg(case))
        s["vertices"] = V.mul_(2.0 ** (seed % 41 - 20))
        s["holes"], s["floaters"] = case["holes"], case["floaters"]
    return s


# ---- one pass ----------------------------------------------------------------------------

def _fit_loss(V):
    """Mean squared distance of the vertices to the sphere of radius 0.3."""
    return (V.norm(dim=1) - 0.3).square().mean()


def run(state):
    kind, be = state["kind"], state["backend"]
    if kind in ("dense", "sparse", "refine"):
        V, F, _ = be.extract_tensor(*state["grid"])
        return V, F
    if kind == "host":
        mesh, _ = be.extract(state["grid"])
        return mesh.vertices, mesh.faces
    if kind == "batch":
        meshes, _ = be.extract_batch(state["grids"])
        return meshes
    if kind == "fit":
        values = state["values"]
        values.grad = None
        V, F = dual_contour(values, *state["where"], backend=be)
        _fit_loss(V).backward()
        return V.detach(), F, values.grad
    if kind == "mesh":
        out, _ = mesh_to_sdf_tensor(be, state["vertices"], state["faces"], state["dims"], state["origin"],
                                    state["spacing"], voxelize_first=state["voxelize"])
        return out
    V, F, _ = postprocess_mesh_tensor(be, state["vertices"], state["faces"], state["holes"], state["floaters"])
    return V, F


def work(case):
    """Bytes: the grid (or the mesh) once in and the result once out. The surface's size is not
    known before a call: a scene crosses about 6 cells per squared resolution (measured on the
    CSG scene, 6.17M at 1024^3; the perturbed sphere 3.1), a vertex is 12 B, a quad 16 B.
    Operations: about 600 per crossed cell (Hermite samples, averaged normals, solve), as
    much again per cell and inner iteration of the refinement, 60 per point-triangle distance."""
    kind = case["kind"]
    if kind == "batch":
        res = _batch_sizes(case)
        points, cells = sum(r ** 3 for r in res), sum(6 * r * r for r in res)
    elif kind == "mesh":
        points, tris = case["res"] ** 3, case["spheres"] * 20 * 4 ** case["subdiv"]
        # a point within 2.5 bins of the surface needs one exact distance at the least
        return {"bytes": 4 * points + 18 * tris, "flops": 60 * min(points, 40 * 6 * case["res"] ** 2)}
    elif "res" in case:
        points, cells = case["res"] ** 3, 3.1 * case["res"] ** 2
    else:
        points = case["nx"] * case["ny"] * case["nz"]
        cells = 6 * points ** (2 / 3)
    if kind == "post":
        return {"bytes": 2 * 28 * cells, "flops": 20 * cells}
    b = 4 * points + 28 * cells + (8 * cells if case.get("triangles") else 0)
    if kind == "fit":
        return {"bytes": b + 4 * points + 12 * cells, "flops": 3 * 600 * cells}
    return {"bytes": b, "flops": 600 * cells * (1 + case.get("outer", 0) * 4)}


# ---- the dense extraction's vertices and their adjoint in 64 bits ------------------------

CORNERS = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))
# (axis, offset of the edge's low corner) of the twelve edges of a cell
EDGES = tuple((a, tuple(0 if d == a else (q >> (0 if d == (a + 1) % 3 else 1)) & 1 for d in range(3)))
              for a in range(3) for q in range(4))
THRESHOLD = 0.01                                # singular values the solve keeps are above it


def _eigenpairs(A):
    """Eigenvalues (n, 3) and eigenvectors (columns, (n, 3, 3)) of symmetric 3x3 matrices by
    cyclic Jacobi rotations, ten sweeps."""
    a = {(i, j): A[:, i, j].clone() for i in range(3) for j in range(i, 3)}
    u = [[torch.full_like(a[0, 0], float(i == j)) for j in range(3)] for i in range(3)]
    for _ in range(10):
        for p, q, r in ((0, 1, 2), (0, 2, 1), (1, 2, 0)):
            apq = a[p, q]
            off = apq != 0
            theta = (a[q, q] - a[p, p]) / (2 * torch.where(off, apq, torch.ones_like(apq)))
            t = torch.where(theta < 0, -1.0, 1.0) / (theta.abs() + (theta * theta + 1).sqrt())
            t = torch.where(off, t, torch.zeros_like(t))
            c = 1 / (t * t + 1).sqrt()
            s = t * c
            pr, qr = (min(p, r), max(p, r)), (min(q, r), max(q, r))
            a[p, p], a[q, q], a[p, q] = a[p, p] - t * apq, a[q, q] + t * apq, torch.zeros_like(apq)
            a[pr], a[qr] = c * a[pr] - s * a[qr], s * a[pr] + c * a[qr]
            for i in range(3):
                u[i][p], u[i][q] = c * u[i][p] - s * u[i][q], s * u[i][p] + c * u[i][q]
    return torch.stack([a[i, i] for i in range(3)], 1), torch.stack([torch.stack(row, 1) for row in u], 1)


class _TruncatedSolve(torch.autograd.Function):
    """x = sum over the eigenpairs of A above THRESHOLD of u (u . r) / lambda."""

    @staticmethod
    def forward(ctx, A, r):
        lam, U = _eigenpairs(A)
        keep = lam.abs() > THRESHOLD
        inv = torch.where(keep, 1 / torch.where(keep, lam.abs(), torch.ones_like(lam)), torch.zeros_like(lam))
        rr = (U * r[:, :, None]).sum(1)
        ctx.save_for_backward(lam, U, keep, inv, rr)
        return (U * (inv * rr)[:, None, :]).sum(2)

    @staticmethod
    def backward(ctx, g):
        lam, U, keep, inv, rr = ctx.saved_tensors
        gg = (U * g[:, :, None]).sum(1)
        p, q = lam[:, :, None], lam[:, None, :]
        kp, kq = keep[:, :, None], keep[:, None, :]
        # divided differences of 1/lambda on the kept, 0 on the truncated eigenvalues
        gap = torch.where(kp == kq, torch.ones_like(p - q), p - q)
        w = torch.where(kp & kq, -inv[:, :, None] * inv[:, None, :], (inv[:, :, None] - inv[:, None, :]) / gap)
        w = torch.where(~kp & ~kq, torch.zeros_like(w), w) * gg[:, :, None] * rr[:, None, :]
        return U @ ((w + w.transpose(1, 2)) / 2) @ U.transpose(1, 2), (U * (inv * gg)[:, None, :]).sum(2)


def _unit(v):
    z = v.square().sum(1, keepdim=True)
    return torch.where(z > 0, v / torch.where(z > 0, z, torch.ones_like(z)).sqrt(), v)


def _vertices(values, dims, sp, org):
    """The vertices of the dense extraction of ``values`` (64 bits, differentiable)."""
    dev = values.device
    n = torch.tensor(dims, device=dev)
    # grid positions are float32 by definition: origin + i * spacing
    pos = [(torch.tensor(o) + torch.arange(m, dtype=torch.float32) * torch.tensor(h)).double().to(dev)
           for m, h, o in zip(dims, sp, org)]
    grid = values.detach().view(dims[2], dims[1], dims[0])

    def some_corner(mask):
        part = (slice(None, -1), slice(1, None))
        out = torch.zeros_like(mask[:-1, :-1, :-1])
        for x, y, z in CORNERS:
            out |= mask[part[z], part[y], part[x]]
        return out

    lin = torch.nonzero((some_corner(grid < 0) & some_corner(grid > 0)).view(-1)).view(-1)
    cx, cy = dims[0] - 1, dims[1] - 1
    cell = torch.stack([lin % cx, lin // cx % cy, lin // (cx * cy)], 1)

    def at(c):
        """The places in the list of active cells of the cells c, and which c are active."""
        inside = ((c >= 0) & (c < n - 1)).all(1)
        key = torch.where(inside, c[:, 0] + cx * (c[:, 1] + cy * c[:, 2]), -1)
        place = torch.searchsorted(lin, key).clamp(max=len(lin) - 1)
        return place, inside & (lin[place] == key)

    f = {o: values[cell[:, 0] + o[0] + dims[0] * (cell[:, 1] + o[1] + dims[1] * (cell[:, 2] + o[2]))] for o in CORNERS}
    lo = torch.stack([pos[d][cell[:, d]] for d in range(3)], 1)
    size = torch.stack([pos[d][cell[:, d] + 1] for d in range(3)], 1) - lo
    crossed, points, normals = {}, {}, {}
    for axis, off in EDGES:
        fa, fb = f[off], f[tuple(1 if d == axis else off[d] for d in range(3))]
        cross = fa * fb <= 0
        t = torch.where(cross, fa, torch.zeros_like(fa)) / torch.where(cross, fa - fb + 1e-16, torch.ones_like(fa))
        w = [t if d == axis else torch.full_like(t, float(off[d])) for d in range(3)]
        g = []
        for d in range(3):                                      # trilinear gradient at the sample
            a, b = (d + 1) % 3, (d + 2) % 3
            s = torch.zeros_like(t)
            for i in (0, 1):
                for j in (0, 1):
                    low, high = [0, 0, 0], [0, 0, 0]
                    low[a], low[b], high[a], high[b], high[d] = i, j, i, j, 1
                    s = s + (f[tuple(high)] - f[tuple(low)]) * (w[a] if i else 1 - w[a]) * (w[b] if j else 1 - w[b])
            g.append(s / size[:, d])
        e = (axis, off)
        crossed[e] = cross[:, None]
        points[e] = lo + size * torch.stack(w, 1)
        normals[e] = torch.where(crossed[e], _unit(torch.stack(g, 1)), torch.zeros_like(lo))
    rows, centre = [], 0.0
    for axis, off in EDGES:
        # averaged over the four cells around the grid edge where all are active and an end of
        # the edge lies inside the grid
        low = cell + torch.tensor(off, device=dev)
        high = low + torch.tensor([d == axis for d in range(3)], device=dev)
        shared = ((low > 0) & (low < n - 1)).all(1) | ((high > 0) & (high < n - 1)).all(1)
        total = torch.zeros_like(lo)
        for other_axis, o in EDGES:
            if other_axis == axis:
                place, active = at(low - torch.tensor(o, device=dev))
                shared = shared & active
                total = total + normals[(axis, o)][place]
        e = (axis, off)
        rows.append((_unit(torch.where(shared[:, None], _unit(total), normals[e])), points[e], crossed[e]))
        centre = centre + points[e] * crossed[e]
    centre = centre / sum(m.double() for _, _, m in rows)
    A, r = 0.0, 0.0
    for normal, point, m in rows:
        A = A + normal[:, :, None] * normal[:, None, :]
        r = r + normal * (normal * (point - centre)).sum(1, keepdim=True)
    return centre + _TruncatedSolve.apply(A, r)


def exact(case, seed):
    """64-bit vertices of the dense kinds and the fit's gradient; whole numbers have no such value.
    The sparse backends, the mesh conversion and the post-pass are defined operation by
    operation in float32 (their decisions included), so their value in 64 bits is another mesh;
    the refinement's in 64 bits takes minutes."""
    kind = case["kind"]
    if kind in ("dense", "host", "batch"):
        Vs = [_vertices(vals.double(), *where) for vals, *where in _grids(case, seed)]
        return [(V, None) for V in Vs] if kind == "batch" else (Vs[0] if kind == "dense" else Vs[0].view(-1), None)
    if kind == "fit":
        (vals, *where), = _grids(case, seed)
        vals = vals.double().requires_grad_(True)
        V = _vertices(vals, *where)
        _fit_loss(V).backward()
        return V.detach(), None, vals.grad
    return None
