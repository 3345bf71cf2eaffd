"""The mark where its tiles change: 256-cell x-tiles of a row or, in batches, four rows a warp,
1024-cell tiles with and without empty chunks, one plane to many; alone and in a batch. Active cells
against numpy, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(2, 2, 2), (33, 8, 9), (34, 9, 3), (65, 32, 2), (256, 33, 40), (257, 34, 7), (258, 16, 30), (96, 200, 180),
         (192, 190, 161), (129, 17, 400), (513, 9, 20), (640, 20, 11), (1000, 8, 9), (1025, 9, 8), (1153, 7, 5), (2300, 9, 4)]


def _grid(dims, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    v = rng.uniform(-1, 1, (nz, ny, nx)).astype(np.float32) * (rng.random((nz, ny, nx)) < 0.7)      # zeros among them
    v[:, : ny // 2] = np.abs(v[:, : ny // 2])                                                          # a quiet half
    return v


def _active(v):
    c = [v[z:v.shape[0] - 1 + z, y:v.shape[1] - 1 + y, x:v.shape[2] - 1 + x] for z in (0, 1) for y in (0, 1) for x in (0, 1)]
    return np.nonzero((np.any([a < 0 for a in c], 0) & np.any([a > 0 for a in c], 0)).ravel())[0]


@pytest.mark.parametrize("dims", SIZES)
def test_alone(dims):
    import torch
    from contouring_b200 import B200DualContouringBackend
    v = _grid(dims, sum(dims))
    be = B200DualContouringBackend(0)
    be.extract_tensor(torch.from_numpy(v.ravel()).cuda(), dims, (0.1,) * 3, (0.0,) * 3)
    cells = be.active_cells()
    be.close()
    assert np.array_equal(cells, _active(v))


def test_batch():
    import torch
    from contouring_b200 import B200DualContouringBackend
    grids = [_grid(d, i) for i, d in enumerate(SIZES)]
    be = B200DualContouringBackend(0)
    one = B200DualContouringBackend(0)
    meshes, _ = be.extract_batch([(torch.from_numpy(v.ravel()).cuda(), d, (0.1,) * 3, (0.0,) * 3) for v, d in zip(grids, SIZES)])
    for (V, F), v, d in zip(meshes, grids, SIZES):
        Va, Fa, _ = one.extract_tensor(torch.from_numpy(v.ravel()).cuda(), d, (0.1,) * 3, (0.0,) * 3)
        assert len(V) == len(_active(v)) and torch.equal(F, Fa)
        assert torch.allclose(V, Va, rtol=0, atol=1e-5, equal_nan=True)       # separately compiled kernels: 1e-4 cell widths
    be.close()
    one.close()
