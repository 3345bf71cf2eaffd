"""The mesh -> SDF band kernel on grids whose spacing is small against the origin, so that points
round to one position: a bin holds more of them than the 15 an axis of even spacing (more than 128
bricks of points, repeats of the full walk among them) and begins far from its nominal first point. Its float operations are the oracle's,
and ties only decide signs, so the values are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _one_column():
    """All 40 x 40 points of a plane at one position, in one bin of 400 bricks; above and below
    the apex of a double cone 40 triangles tie."""
    a = 2 * np.pi * np.arange(40) / 40
    ring = np.stack([np.round(64 * np.cos(a)) / 8, np.round(64 * np.sin(a)) / 8, 0 * a], 1)
    V = np.concatenate([ring + [1e6, 1e6, -1.0], [[1e6, 1e6, 0.128], [1e6, 1e6, -2.0]]])
    i, j = np.arange(40), (np.arange(40) + 1) % 40
    F = np.concatenate([np.stack([i, j, 0 * i + 40], 1), np.stack([j, i, 0 * i + 41], 1)])
    return V, F, (40, 40, 64), (0.0005, 0.0005, 0.004), (1e6, 1e6, 0.0)


def _sheet(dims, sp, org, pitch):
    """A wavy sheet across the grid's middle in z, facets of `pitch` a side."""
    n = [int(np.ceil(d * h / pitch)) + 2 for d, h in zip(dims, sp)]
    x, y = np.meshgrid(np.arange(n[0] + 1) * pitch - pitch, np.arange(n[1] + 1) * pitch - pitch, indexing="ij")
    z = dims[2] * sp[2] * (0.5 + 0.15 * np.sin(3 * x / (dims[0] * sp[0])) * np.cos(4 * y / (dims[1] * sp[1])))
    V = np.stack([x + org[0], y + org[1], z + org[2]], 2).reshape(-1, 3)
    at = np.arange(V.shape[0]).reshape(n[0] + 1, n[1] + 1)
    a, b, c, d = at[:-1, :-1].ravel(), at[1:, :-1].ravel(), at[1:, 1:].ravel(), at[:-1, 1:].ravel()
    return V, np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1)]), dims, sp, org


# projected coordinates of a scan; every axis bunched
SCENES = {"one_column": _one_column,
          "scan": lambda: _sheet((256, 512, 64), (0.005,) * 3, (5e5, 4.2e6, 0.0), 0.05),
          "cube64": lambda: _sheet((64, 64, 64), (0.001,) * 3, (1e6, 1e6, 1e6), 0.0625),
          "cube100": lambda: _sheet((100, 100, 100), (0.01,) * 3, (1e7, 1e7, 1e7), 1.0)}


@pytest.mark.parametrize("name", sorted(SCENES))
def test_bunched_positions_equal_oracle(name):
    import oracle as O
    import torch
    from contouring_b200 import B200DualContouringBackend, mesh_to_sdf_tensor
    V, F, dims, sp, org = SCENES[name]()
    V, F = V.astype(np.float32), F.astype(np.int32)
    be = B200DualContouringBackend(0)
    out, _ = mesh_to_sdf_tensor(be, torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), dims, org, sp)
    ref, _ = O.mesh_to_sdf(V, F, dims, org, sp)
    got = out.cpu().numpy()
    be.close()
    assert np.array_equal(got, ref), "%d of %d values differ" % (int((got != ref).sum()), got.size)
