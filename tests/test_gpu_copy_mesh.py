"""dcb_copy_mesh_device: one kernel into arrays of the mesh's own GPU, the copy engine into any other
device-accessible memory (an array on another GPU may not be mapped for this one's kernels). Managed
memory stands for the second kind: a kernel could store there too, so both routes are safe to run."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["own", "managed", "odd"])
def test_route_and_contents(where):
    import torch
    from contouring_b200 import B200DualContouringBackend, _lib, synth
    be = B200DualContouringBackend(0)
    V, F, _ = be.extract_tensor(*(g.cuda() if torch.is_tensor(g) else g for g in synth.csg(24, seed=1)))
    sizes = (V.numel() * 4, F.numel() * 4)
    cudart = ctypes.CDLL("libcudart.so.12")
    keep = []
    if where == "managed":
        ptrs = []
        for n in sizes:
            p = ctypes.c_void_p()
            assert cudart.cudaMallocManaged(ctypes.byref(p), ctypes.c_size_t(n), 1) == 0
            ptrs.append(p.value)
    else:
        keep = [torch.zeros(n // 4 + 4, dtype=torch.int32, device="cuda") for n in sizes]
        ptrs = [t.data_ptr() + (4 if where == "odd" else 0) for t in keep]
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        _lib.check(be._L.dcb_copy_mesh_device(be._h, ptrs[0], ptrs[1], None), be._h)
        torch.cuda.synchronize()
    names = " ".join(e.key for e in prof.key_averages())
    assert ("k_copy_mesh" in names) == (where == "own"), names
    for p, ref in zip(ptrs, (V, F)):
        got = np.empty(ref.shape, np.uint32)
        assert cudart.cudaMemcpy(ctypes.c_void_p(got.ctypes.data), ctypes.c_void_p(p), ctypes.c_size_t(got.nbytes), 4) == 0
        assert np.array_equal(got, ref.cpu().numpy().view(np.uint32))
    if where == "managed":
        for p in ptrs:
            cudart.cudaFree(ctypes.c_void_p(p))
    be.close()
