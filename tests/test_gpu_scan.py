"""The exclusive scan behind the extraction at the sizes where its form changes (one block up to
16,384 counts, two launches up to 2,048 blocks of 2,048, three beyond), through the entry point
that scans a grid's row counts: every active cell in ascending order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 16384, 16385, (1 << 21) - 1, 2048 * 2048 + 2])
def test_active_cells_across_scan_forms(rows):
    import torch
    from contouring_b200 import B200DualContouringBackend
    # one cell wide: cell row (j, k) is active where the sign, a function of j, changes from j to j + 1
    nz = 1 if rows < 1 << 21 else 3
    ny = rows // nz
    rng = np.random.default_rng(rows)
    sign = rng.integers(0, 2, ny + 1) * 2 - 1
    vals = np.tile(np.repeat(sign.astype(np.float32), 2), nz + 1)   # nx = 2
    be = B200DualContouringBackend(0)
    V, F, st = be.extract_tensor(torch.from_numpy(vals).cuda(), (2, ny + 1, nz + 1), (1e-3,) * 3, (0.0,) * 3)
    cells = be.active_cells()
    be.close()
    one = np.nonzero(sign[1:] != sign[:-1])[0]
    assert np.array_equal(cells, np.concatenate([one + ny * k for k in range(nz)])) and len(V) == len(cells)
