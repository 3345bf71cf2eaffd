"""The refinement's inner loop where its team sizes change (cells with a few, some tens and hundreds
of spheres in one grid) and its closest-point search where it leaves a thread's budget (points at
equal distance from many triangles), against the oracle. Tolerance: the output's float rounding of
coordinates up to 0.5 (3e-8) in cell widths of 1/23, and the oracle's own FP64 noise, below 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(n, half):
    """Euclidean distance to a cube: a corner's cell takes the spheres of a whole octant, an
    edge's those of a column."""
    import torch
    ax = np.linspace(-0.5, 0.5, n)
    q = np.abs(np.stack(np.meshgrid(ax, ax, ax, indexing="ij"), -1)) - half
    d = np.linalg.norm(np.maximum(q, 0), axis=-1) + np.minimum(q.max(-1), 0)
    step = float(np.float32(1.0 / (n - 1)))
    return torch.from_numpy(d.astype(np.float32).transpose(2, 1, 0).reshape(-1).copy()), (n,) * 3, (step,) * 3, (-0.5,) * 3


@pytest.mark.parametrize("name", ["corners", "centre"])
def test_teams_match_oracle(name):
    import oracle as O
    from contouring_b200 import B200DualContouringBackend, ContouringMethod, ContouringOptions, synth
    vals, dims, sp, org = _box(24, 0.22) if name == "corners" else synth.sphere(25, radius=0.4)
    o = ContouringOptions()
    o.method = ContouringMethod.Ours
    o.outer_iters = 2
    o.batch_size = 24 ** 3
    be = B200DualContouringBackend(0, o)
    V, F, _ = be.extract_tensor(vals.cuda(), dims, sp, org)
    r = O.ours(vals.numpy(), dims, sp, org, outer_iters=2, batch_size=24 ** 3)
    be.close()
    assert np.array_equal(F.cpu().numpy(), r["F"])
    assert np.abs(V.cpu().numpy().astype(np.float64) - r["V"]).max() <= 1e-5 * sp[0]
