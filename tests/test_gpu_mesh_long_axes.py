"""mesh -> SDF on grids that are very long along one axis (more tiles than a launch has blocks in its
second and third dimension), with a mesh at the far end. The float operations are the oracle's, so
the values are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis,n", [(0, 1572900), (1, 1572840), (1, 1572841), (1, 1600003), (2, 1048561), (2, 1572900)])
def test_long_axis_equals_oracle(axis, n):
    import oracle as O
    import torch
    from contouring_b200 import B200DualContouringBackend, mesh_to_sdf_tensor, synth
    V, F = synth.icosphere_scene(1, 1, seed=3)
    V = (V - V.min(0)) / (V.max(0) - V.min(0)).max()                 # within [0, 1]^3
    dims, sp = [3, 4, 5], (0.0625, 0.0625, 0.0625)
    dims[axis] = n
    V = V * 0.125
    V[:, axis] = V[:, axis] * 24 + (n - 60) * sp[axis]
    V = V.astype(np.float32)
    be = B200DualContouringBackend(0)
    out, _ = mesh_to_sdf_tensor(be, torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), dims, (0.0, 0.0, 0.0), sp)
    ref, _ = O.mesh_to_sdf(V, F, dims, (0.0, 0.0, 0.0), sp)
    got = out.cpu().numpy()
    be.close()
    assert np.array_equal(got, ref), "%d of %d values differ" % (int((got != ref).sum()), got.size)
