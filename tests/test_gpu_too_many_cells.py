"""Grids with 2^32 and more active cells, which 32-bit ranks do not hold: refused, by a fresh handle and
by one with the buffers of an earlier call, and the handle works on. Every cell of a checkerboard of
signs is active: 2^32 of them in 4,194,304 segments (the two-launch scan), 1,639^3 in more."""
import pytest

pytestmark = pytest.mark.gpu


def _checkerboard(dims):
    import torch
    nx, ny, nz = dims
    i, j = torch.arange(nx, device="cuda"), torch.arange(ny, device="cuda")
    plane = (((i[None, :] + j[:, None]) & 1) * 2 - 1).float()
    v = torch.empty((nz, ny, nx), device="cuda")
    v[0::2] = plane
    v[1::2] = -plane
    return v.view(-1)


@pytest.mark.parametrize("dims", [(1025, 2049, 2049), (1640, 1640, 1640)])
def test_more_active_cells_than_ranks(dims):
    import torch
    from contouring_b200 import B200DualContouringBackend, _lib, synth
    small = [g.cuda() if torch.is_tensor(g) else g for g in synth.sphere(40, 0.3)]
    be = B200DualContouringBackend(0)
    v = _checkerboard(dims)
    with pytest.raises(_lib.DcbError) as e:
        be.extract_tensor(v, dims, (1.0,) * 3, (0.0,) * 3)
    assert "2^31" in str(e.value)
    V, F, _ = be.extract_tensor(*small)
    with pytest.raises(_lib.DcbError):
        be.extract_tensor(v, dims, (1.0,) * 3, (0.0,) * 3)
    V2, F2, _ = be.extract_tensor(*small)
    assert torch.equal(V, V2) and torch.equal(F, F2) and len(V) > 0
    be.close()
