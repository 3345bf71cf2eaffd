"""mesh -> SDF with more bin entries than 32 bits count: 64^3 bins, each of which lists every one of
16,500 triangles across the whole grid (4,325,376,000 entries, 30,408,704 modulo 2^32). Refused, and
the handle works on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_entries_beyond_32_bits_are_refused():
    import torch
    from contouring_b200 import B200DualContouringBackend, _lib, mesh_to_sdf_tensor, synth
    n = 16500
    V = np.array([[-9, -9, -9], [9, -9, 9], [-9, 9, 9], [9, 9, 9]], np.float32)
    F = np.tile(np.array([[0, 1, 2], [0, 3, 1]], np.int32), (n // 2, 1))
    be = B200DualContouringBackend(0)
    with pytest.raises(_lib.DcbError) as e:
        mesh_to_sdf_tensor(be, torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), (512,) * 3, (0.0,) * 3, (1 / 512,) * 3)
    assert "entries" in str(e.value)
    V, F = synth.icosphere_scene(1, 1, seed=3)
    dims, sp, org = synth.mesh_grid(V, 24)
    out, _ = mesh_to_sdf_tensor(be, torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), dims, org, sp)
    assert bool((out < 0).any()) and bool((out > 0).any())
    be.close()
