"""The mesh -> SDF band kernel where its walk over a bin's triangles can go wrong: more triangles
tied at a point than it collects, lists longer than a CTA holds, bins of uneven sides, squared
distances at the tie rule's absolute floor. Its float operations are the oracle's, and ties
only decide signs, so the values are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fan(n):
    """A closed double cone with n triangles at each apex."""
    a = 2 * np.pi * np.arange(n) / n
    ring = np.stack([0.3 * np.cos(a), 0.3 * np.sin(a), 0 * a], 1)
    V = np.concatenate([ring, [[0, 0, 0.25], [0, 0, -0.25]]]).astype(np.float32)
    i, j = np.arange(n), (np.arange(n) + 1) % n
    F = np.concatenate([np.stack([i, j, 0 * i + n], 1), np.stack([j, i, 0 * i + n + 1], 1)]).astype(np.int32)
    return V, F


def _scene(name):
    from contouring_b200 import synth
    if name == "apex_of_7":                         # as many as are collected
        V, F = _fan(7)
        return V, F, synth.mesh_grid(V, 40)
    if name == "apex_of_40":                        # more: the full walk
        V, F = _fan(40)
        return V, F, synth.mesh_grid(V, 40)
    if name == "stacked":                           # every triangle nine times
        V, F = synth.icosphere_scene(1, 1, seed=6)
        return V, np.tile(F, (9, 1)), synth.mesh_grid(V, 32)
    if name == "long_lists":                        # hundreds of distinct triangles around a bin
        V, F = synth.icosphere_scene(6, 4, seed=7)
        return V, F, synth.mesh_grid(V, 24)
    if name == "uneven_bins":                       # bins of 9 to 15 points a side
        V, F = synth.icosphere_scene(3, 2, seed=8)
        _, sp, org = synth.mesh_grid(V, 31)
        return V, F, ((27, 31, 15), (sp[0] * 30 / 26, sp[1], sp[2] * 30 / 14), org)
    if name == "tie_floor":                         # squared distances near 1e-8 * 1e-5
        V, F = synth.icosphere_scene(2, 2, seed=9)
        V = (V * np.float32(2e-5)).astype(np.float32)
        return V, F, synth.mesh_grid(V, 40)
    raise KeyError(name)


@pytest.mark.parametrize("name", ["apex_of_7", "apex_of_40", "stacked", "long_lists", "uneven_bins", "tie_floor"])
def test_band_equals_oracle(name):
    import oracle as O
    import torch
    from contouring_b200 import B200DualContouringBackend, mesh_to_sdf_tensor
    V, F, (dims, sp, org) = _scene(name)
    be = B200DualContouringBackend(0)
    out, _ = mesh_to_sdf_tensor(be, torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), dims, org, sp)
    ref, _ = O.mesh_to_sdf(V, F, dims, org, sp)
    got = out.cpu().numpy()
    be.close()
    assert np.array_equal(got, ref), "%d of %d values differ" % (int((got != ref).sum()), got.size)
