"""Device memory of the refinement per grid point, which limits the grids it takes: eight 32-bit and
two 64-bit arrays over the points (48 bytes), the sort's alternate keys, values and
counts (13), an eighth of headroom, and 5 bytes for the extraction's words and the few cells."""
import pytest

pytestmark = pytest.mark.gpu


def test_bytes_per_point():
    import torch
    from contouring_b200 import B200DualContouringBackend, ContouringMethod, ContouringOptions, synth
    vals, dims, sp, org = synth.sphere(256, 0.03)
    vals = vals.cuda()
    o = ContouringOptions()
    o.method = ContouringMethod.Ours
    o.outer_iters, o.inner_iters = 1, 1
    torch.cuda.synchronize()
    be = B200DualContouringBackend(0, o)
    before = torch.cuda.mem_get_info()[0]
    be.extract_tensor(vals, dims, sp, org)
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    be.close()
    assert used <= ((48 + 13) * 9 / 8 + 5) * vals.numel(), used / vals.numel()
