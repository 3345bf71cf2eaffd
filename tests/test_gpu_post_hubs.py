"""The mesh post-pass around hub vertices, whose edge uses a block sorts: sizes at the edges of its
network (powers of two, the largest), runs of one, two, three and more uses, many hubs at once;
against the oracle, bit for bit. And a fan of 8,000 uses beside the sorted form, which serves one of
8,400: as fast within a factor of two (a walk over all pairs of uses takes ten times as long)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hubs(sizes, repeats=1):
    """A fan of n quads (apex, rim, mid, rim) for every n: 2 n uses at an apex of small index, its outer
    rims left open; every seventh quad of the first fan `repeats` times more."""
    V, F = [[3.0 * c, 0.0, 0.5] for c in range(len(sizes))], []
    for c, n in enumerate(sizes):
        base = len(V)
        a = 2 * np.pi * np.arange(n + 1) / (n + 2)
        V += np.stack([3.0 * c + np.cos(a), np.sin(a), 0 * a], 1).tolist()
        V += np.stack([3.0 * c + 1.2 * np.cos(a + 0.01), 1.2 * np.sin(a + 0.01), 0 * a - 0.1], 1).tolist()
        F += [[c, base + i, base + n + 1 + i, base + i + 1] for i in range(n)]
    F += F[:sizes[0]:7] * repeats
    return np.array(V, np.float32), np.array(F, np.int32)


@pytest.mark.parametrize("sizes,repeats", [((17,), 1), ((32, 33, 16, 64, 65), 2), ((256, 255, 257, 100), 3), ((2048, 2049), 5),
                                           ((4096,), 0), ((40,) * 700, 1)])
@pytest.mark.parametrize("flags", [(True, True), (False, True), (True, False)])
def test_hubs_equal_oracle(sizes, repeats, flags):
    import oracle as O
    import torch
    from contouring_b200 import B200DualContouringBackend, postprocess_mesh_tensor
    V, F = _hubs(sizes, repeats)
    be = B200DualContouringBackend(0)
    Vg, Fg, _ = postprocess_mesh_tensor(be, torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), *flags)
    Vo, Fo, _ = O.postprocess_mesh(V, F, *flags)
    be.close()
    assert np.array_equal(Fg.cpu().numpy(), Fo)
    assert np.array_equal(Vg.cpu().numpy().view(np.uint32), Vo.view(np.uint32))


def test_large_hub_takes_no_longer_than_sorted():
    import torch
    from contouring_b200 import B200DualContouringBackend, postprocess_mesh_tensor
    be = B200DualContouringBackend(0)

    def best(n):
        V, F = (torch.from_numpy(x).cuda() for x in _hubs((n,), 0))
        times = []
        for _ in range(8):
            torch.cuda.synchronize()
            t = time.perf_counter()
            postprocess_mesh_tensor(be, V, F, True, True)
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t)
        return min(times)

    block, sort = best(4000), best(4200)
    be.close()
    assert block < 2 * sort, (block, sort)
