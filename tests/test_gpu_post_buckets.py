"""The mesh post-pass where a vertex has more edge uses than a thread compares (32), than a block
compares (8192: the sorted form), and where welding meets one key many times; against the oracle,
bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fans(n, copies):
    """`copies` fans of n quads (apex, rim, mid, rim) about apexes of smallest indices, the last rim
    left open; one quad doubled (a run of four uses)."""
    V, F = [], []
    for c in range(copies):
        V.append([3.0 * c, 0.0, 0.5])
    for c in range(copies):
        base = copies + c * 2 * (n + 1)
        a = 2 * np.pi * np.arange(n + 1) / (n + 2)
        rim = np.stack([3.0 * c + np.cos(a), np.sin(a), 0 * a], 1)
        mid = np.stack([3.0 * c + 1.2 * np.cos(a + 0.01), 1.2 * np.sin(a + 0.01), 0 * a - 0.1], 1)
        V += rim.tolist() + mid.tolist()
        F += [[c, base + i, base + n + 1 + i, base + i + 1] for i in range(n)]
    F.append(F[-1])
    return np.array(V, np.float32), np.array(F, np.int32)


@pytest.mark.parametrize("n,copies", [(15, 3), (16, 3), (17, 3), (300, 2), (4095, 2), (4200, 2)])
@pytest.mark.parametrize("flags", [(True, True), (False, True), (True, False)])
def test_fans(n, copies, flags):
    import oracle as O
    import torch
    from contouring_b200 import B200DualContouringBackend, postprocess_mesh_tensor
    V, F = _fans(n, copies)
    V = np.concatenate([V, V[:1].repeat(50, 0)])           # 50 more of one point
    F = np.concatenate([F, [[len(V) - 1, 5, 6, 7]]]).astype(np.int32)
    be = B200DualContouringBackend(0)
    Vg, Fg, st = postprocess_mesh_tensor(be, torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), *flags)
    Vo, Fo, ost = O.postprocess_mesh(V, F, *flags)
    assert np.array_equal(Fg.cpu().numpy(), Fo)
    assert np.array_equal(Vg.cpu().numpy().view(np.uint32), Vo.view(np.uint32))
    be.close()
