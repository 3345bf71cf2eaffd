"""The mesh -> SDF band kernel on grids whose spacing is small against the origin, so that points
round to one position and a bin holds more of them than the 15 an axis of even spacing: more than
128 bricks of points, repeats of the full walk among them. Its float operations are the oracle's,
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


SCENES = {"one_column": _one_column}


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
