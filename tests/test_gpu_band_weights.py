"""The mesh -> SDF band's sign where the summed normals have no side: a triangle whose closest point is a
corner with an angle of 0 has weight 0 there (the value is positive), and areas whose squares overflow
give a normalised sum of 0. The band's float operations are the oracle's, so the values are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(name):
    from contouring_b200 import synth
    if name.startswith("slivers"):                  # third corners a few ulps off the first edges
        at = float(name[7:])
        r = np.random.default_rng(int(at))
        a, d = r.uniform(0, 1, (60, 3)), r.normal(0, 0.3, (60, 3))
        V = np.stack([a, a + d, a + d * r.uniform(0, 1, (60, 1))], 1).reshape(-1, 3) + at
        return V, np.arange(180).reshape(-1, 3), 1.0, at
    V, F = synth.icosphere_scene(2, 2, seed=4)
    if name.startswith("fives"):                    # every triangle five times: their sum overflows
        F = np.tile(F, (5, 1))
    return (V - V.min(0)) / (V.max(0) - V.min(0)).max(), F, float(name[5:]), 0.0


@pytest.mark.parametrize("name", ["slivers0", "slivers64", "slivers256", "slivers1024", "scale1e8", "scale1e9", "scale1e10",
                                  "scale1e12", "fives1e10", "fives12e9", "fives14e9", "fives2e10"])
def test_sign_equals_oracle(name):
    import oracle as O
    import torch
    from contouring_b200 import B200DualContouringBackend, mesh_to_sdf_tensor
    V, F, unit, at = _scene(name)
    V, F = (V * unit).astype(np.float32), F.astype(np.int32)
    dims, sp, org = (33, 30, 36), (0.04 * unit,) * 3, (-0.1 * unit + at,) * 3
    be = B200DualContouringBackend(0)
    out, _ = mesh_to_sdf_tensor(be, torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), dims, org, sp)
    ref, _ = O.mesh_to_sdf(V, F, dims, org, sp)
    got = out.cpu().numpy()
    be.close()
    assert np.array_equal(got, ref), "%d of %d values differ" % (int((got != ref).sum()), got.size)
