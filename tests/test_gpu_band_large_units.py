"""The mesh -> SDF band in units where the barycentric coordinates' products overflow, so that some float
distances come out too long: no distance is bounded by a triangle's there. The band's float
operations are the oracle's, so the values are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unit", [1e7, 1e8, 1e9, 1e10, 5e10, 1e11, 1e13, 1e15])
@pytest.mark.parametrize("seed", [34, 35])
def test_large_units_equal_oracle(unit, seed):
    import oracle as O
    import torch
    from contouring_b200 import B200DualContouringBackend, mesh_to_sdf_tensor, synth
    V, F = synth.icosphere_scene(3, 1, seed=seed)
    V = (V * np.float32(unit)).astype(np.float32)
    dims, sp, org = synth.mesh_grid(V, 34)
    be = B200DualContouringBackend(0)
    out, _ = mesh_to_sdf_tensor(be, torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), dims, org, sp)
    ref, _ = O.mesh_to_sdf(V, F, dims, org, sp)
    got = out.cpu().numpy()
    be.close()
    assert np.array_equal(got, ref), "%d of %d values differ" % (int((got != ref).sum()), got.size)
