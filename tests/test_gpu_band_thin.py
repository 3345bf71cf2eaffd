"""The mesh -> SDF band with thin triangles, whose float normals are off by a good angle: they bound no
distance. Slivers with the third corner within 1e-4, 1e-5 and 1e-6 of the first edge. The band's
float operations are the oracle's, so the values are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("digits", [4, 5, 6])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_slivers_equal_oracle(digits, seed):
    import oracle as O
    import torch
    from contouring_b200 import B200DualContouringBackend, mesh_to_sdf_tensor
    r = np.random.default_rng(seed)
    a, d = r.uniform(0, 1, (150, 3)), r.normal(0, 0.3, (150, 3))
    c = a + d * r.uniform(0, 1, (150, 1)) + r.normal(0, 10.0 ** -digits, (150, 3))
    V, F = np.stack([a, a + d, c], 1).reshape(-1, 3).astype(np.float32), np.arange(450, dtype=np.int32).reshape(-1, 3)
    dims, sp, org = (53, 48, 57), (0.025,) * 3, (-0.1,) * 3
    be = B200DualContouringBackend(0)
    out, _ = mesh_to_sdf_tensor(be, torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), dims, org, sp)
    ref, _ = O.mesh_to_sdf(V, F, dims, org, sp)
    got = out.cpu().numpy()
    be.close()
    assert np.array_equal(got, ref), "%d of %d values differ" % (int((got != ref).sum()), got.size)
