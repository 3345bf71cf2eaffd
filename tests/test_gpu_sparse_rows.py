"""The sparse backends' marking where rows change their share of a warp (up to 8, 16 and 32 cell
words a row, several segments a row) and of a block (point words against its threads), against the
oracle: identical vertices and faces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [2, 33, 257, 258, 513, 514, 1025, 1026, 4200])
def test_row_lengths(nx):
    import oracle as O
    import torch
    from contouring_b200 import B200SparseDualContouringBackend
    dims, sp, org = (nx, 7, 6), (0.01, 0.01, 0.01), (0.0, 0.0, 0.0)
    rng = np.random.default_rng(nx)
    z, y, x = np.meshgrid(np.arange(6), np.arange(7), np.arange(nx), indexing="ij")
    v = (0.01 * (y - 3.0 + 1.5 * np.sin(0.05 * x) + 0.2 * z) + rng.uniform(-2e-3, 2e-3, x.shape)).astype(np.float32).ravel()
    for brick in (3, 8):
        be = B200SparseDualContouringBackend(brick_size=brick)
        V, F, st = be.extract_tensor(torch.from_numpy(v).cuda(), dims, sp, org)
        r = O.sparse_extract(v, dims, sp, org, brick_size=brick, mvdc=False, normal_mode=0)
        be.close()
        assert np.array_equal(F.cpu().numpy(), r["F"])
        assert np.array_equal(V.cpu().numpy().view(np.uint32), r["V"].view(np.uint32))
