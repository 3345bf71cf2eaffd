"""The refinement's inner loop with more cells than the GPU's blocks hold at once, so that freed
slots are filled again (27,486 cells; a full GPU holds 16,576), against the oracle. Tolerance as
for the smaller scenes: the output's float rounding of coordinates up to 0.5 (3e-8) in cell widths
of 1/127 and the oracle's own FP64 noise, below 1e-5 of a cell."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inner_iters", [2])
def test_refilled_slots_match_oracle(inner_iters):
    import oracle as O
    from contouring_b200 import B200DualContouringBackend, ContouringMethod, ContouringOptions, synth
    vals, dims, sp, org = synth.rbf_sphere(128)
    o = ContouringOptions()
    o.method = ContouringMethod.Ours
    o.outer_iters, o.inner_iters, o.batch_size = 1, inner_iters, 1
    be = B200DualContouringBackend(0, o)
    V, F, _ = be.extract_tensor(vals.cuda(), dims, sp, org)
    r = O.ours(vals.numpy(), dims, sp, org, outer_iters=1, inner_iters=inner_iters, batch_size=1)
    be.close()
    assert np.array_equal(F.cpu().numpy(), r["F"])
    assert np.abs(V.cpu().numpy().astype(np.float64) - r["V"]).max() <= 1e-5 * sp[0]
