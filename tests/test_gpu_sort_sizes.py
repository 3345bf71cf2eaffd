"""The stable sort behind the mesh post-pass where it changes form (one block up to 8,192 items) and
cycle ranking where it does (one block up to 16,384 boundary edges): open strips whose boundary
edges number just below and above, against the oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edges", [6, 62, 4094, 8190, 8192, 8194, 16384, 16386])
def test_strips(edges):
    import oracle as O
    import torch
    from contouring_b200 import B200DualContouringBackend, postprocess_mesh_tensor
    n = edges // 2 - 1                                   # quads of a strip: 2n + 2 boundary edges, one cycle
    rng = np.random.default_rng(edges)
    x = np.arange(n + 1)
    V = np.concatenate([np.stack([x, 0 * x, 0 * x], 1), np.stack([x, 0 * x + 1, 0.1 * x], 1)]).astype(np.float32)
    F = np.stack([x[:-1], x[1:], n + 2 + x[:-1], n + 1 + x[:-1]], 1)
    order = rng.permutation(2 * (n + 1))                 # vertices and faces in no order
    V, F = V[np.argsort(order)], order[F][rng.permutation(n)].astype(np.int32)
    be = B200DualContouringBackend(0)
    Vg, Fg, st = postprocess_mesh_tensor(be, torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), True, True)
    Vo, Fo, ost = O.postprocess_mesh(V, F, True, True)
    be.close()
    assert st.boundary_edges == edges
    assert np.array_equal(Fg.cpu().numpy(), Fo)
    assert np.array_equal(Vg.cpu().numpy().view(np.uint32), Vo.view(np.uint32))
