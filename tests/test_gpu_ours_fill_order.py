"""The refinement's random fill at the size from which it is sorted (98,304 points), one more, and all
points but one, against the oracle, which sorts all keys. Tolerance: the output's float rounding of
coordinates up to 0.5 (3e-8) in cell widths of 1/51 and the oracle's own FP64 noise, below 1e-5 of
a cell; another set of spheres moves vertices by far more."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fill", [98304, 98305, None])
def test_fill_matches_oracle(fill):
    import oracle as O
    from contouring_b200 import B200DualContouringBackend, ContouringMethod, ContouringOptions, synth
    vals, dims, sp, org = synth.sphere(52, radius=0.3)
    near = int((vals.double().abs() < 3 * math.sqrt(sum(h * h for h in sp))).sum())
    batch = near + fill if fill else 52 ** 3 - 1
    o = ContouringOptions()
    o.method = ContouringMethod.Ours
    o.outer_iters, o.inner_iters, o.batch_size = 2, 4, batch
    be = B200DualContouringBackend(0, o)
    V, F, _ = be.extract_tensor(vals.cuda(), dims, sp, org)
    r = O.ours(vals.numpy(), dims, sp, org, outer_iters=2, inner_iters=4, batch_size=batch)
    be.close()
    assert np.array_equal(F.cpu().numpy(), r["F"])
    assert np.abs(V.cpu().numpy().astype(np.float64) - r["V"]).max() <= 1e-5 * sp[0]
