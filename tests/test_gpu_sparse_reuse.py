"""The sparse backends on the buffers of an earlier call (everything launched with the count read on
the device): after a larger grid, after a smaller one (run again with buffers for the count; or
enough cells but more faces than before), and on a grid without active cells."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("multi", [False, True])
@pytest.mark.parametrize("before", ["csg96", "sphere20", "empty", "noise"])
def test_reused_equals_fresh(before, multi):
    from contouring_b200 import B200SparseDualContouringBackend, synth
    grids = {"csg96": lambda: synth.csg(96, seed=4), "sphere20": lambda: synth.sphere(20, 0.3),
             "empty": lambda: synth.constant(16, 1.0),
             "noise": lambda: synth.noise((40, 40, 40), seed=5, scale=0.04)}     # near zero: many cells, few faces

    def run(be, grid):
        V, F, st = be.extract_tensor(grid[0].cuda(), *grid[1:])
        d = st.as_dict()
        return V.cpu().numpy(), F.cpu().numpy(), be.active_cells(), {k: v for k, v in d.items() if not k.endswith("_ms")}

    for grid in (synth.thin_shell(48, seed=1), synth.csg(64, seed=2), grids["empty"]()):
        fresh = B200SparseDualContouringBackend(multi_vertex_cells=multi)
        warm = B200SparseDualContouringBackend(multi_vertex_cells=multi)
        ref = run(fresh, grid)
        run(warm, grids[before]())
        for _ in range(2):
            got = run(warm, grid)
            for a, b in zip(ref[:3], got[:3]):
                assert np.array_equal(a, b)
            assert ref[3] == got[3]
        fresh.close()
        warm.close()
