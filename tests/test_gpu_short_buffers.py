"""Single-operator calls on a device buffer that ends before its field does."""
import ctypes

import numpy as np
import pytest

from afmibins_gb300 import capi

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _alloc(nbytes):
    """An allocation of its own (torch's are cut from larger ones)."""
    torch.zeros(1, device="cuda")  # makes the device's context current
    cu, p = ctypes.CDLL("libcuda.so.1"), ctypes.c_uint64(0)
    assert cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(nbytes)) == 0
    return cu, p


@pytest.mark.parametrize("short_out", [False, True])
def test_short_device_buffer_is_refused(short_out):
    """Half a field: the call returns an error, as the copy of such a buffer does,
    instead of running a kernel over its end (the field is far below the 2 MB that
    the device maps at a time). The solver goes on working."""
    with capi.Solver(32) as sv:
        N = sv.ncell
        cu, small = _alloc(N * 4)
        full = torch.full((N,), 3.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        half, whole = small.value, capi.ptr(full)
        try:
            out, inp = (half, whole) if short_out else (whole, half)
            assert sv.lib.afmib_lap_apply(sv.h, out, inp) == 2  # AFMIB_ERR_CUDA
            assert bool((full == 3.0).all())
            b = np.random.default_rng(0).standard_normal(N)
            ref, dev = np.zeros(N), torch.from_numpy(b).cuda()
            torch.cuda.synchronize()
            assert sv.lib.afmib_lap_apply(sv.h, capi.ptr(ref), capi.ptr(b)) == 0
            assert sv.lib.afmib_lap_apply(sv.h, whole, capi.ptr(dev)) == 0
            assert np.array_equal(full.cpu().numpy(), ref)
        finally:
            assert cu.cuMemFree_v2(small) == 0
