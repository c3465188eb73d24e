"""fp_solve_permeability where the memory of the lockstep's two siblings is not
there: the current device pool is one of 32 MB for the call, and the load cases
are solved one at a time, with the K and iterations they have alone."""
import ctypes as C
import math

import numpy as np
import pytest

from fft_method_test_gb300 import geometry as G

pytestmark = pytest.mark.gpu


class _Props(C.Structure):  # CUmemPoolProps
    _fields_ = [("alloc_type", C.c_int), ("handle_types", C.c_int), ("location_type", C.c_int),
                ("location_id", C.c_int), ("security", C.c_void_p), ("max_size", C.c_size_t),
                ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_no_memory_for_the_siblings(gpu_lib, precision):
    from fft_method_test_gb300 import _capi
    from fft_method_test_gb300.permeability import PermeabilityProblem

    cu = C.CDLL("libcuda.so.1")
    mask = G.gaussian_field(128, 5.0, 0.45, seed=8)
    with PermeabilityProblem(mask.shape, precision=precision) as p:
        p.set_geometry(mask)
        K, st = p.solve_permeability(1e-12, 20)
        cases = [p.solve_load_case(np.eye(3)[c], 1e-12, 20) for c in range(3)]
        dev, old, small = C.c_int(), C.c_void_p(), C.c_void_p()
        assert cu.cuCtxGetDevice(C.byref(dev)) == 0
        assert cu.cuDeviceGetMemPool(C.byref(old), dev) == 0
        props = _Props(alloc_type=1, location_type=1, location_id=dev.value, max_size=32 << 20)
        if cu.cuMemPoolCreate(C.byref(small), C.byref(props)) != 0:
            pytest.skip("no bounded memory pools")
        try:
            assert cu.cuDeviceSetMemPool(dev, small) == 0
            K2, st2 = p.solve_permeability(1e-12, 20)
            with pytest.raises(_capi.FpError):  # the block is asked for by name: its failure is reported
                p.solve_permeability(1e-12, 20, block=True)
        finally:
            assert cu.cuDeviceSetMemPool(dev, old) == 0
            cu.cuMemPoolDestroy(small)
        K3, _ = p.solve_permeability(1e-12, 20)
    assert np.array_equal(K, K2) and np.array_equal(K, K3)
    for c in range(3):
        assert np.array_equal(K2[:, c], p.mu * cases[c][0])
        assert st2[c]["iterations"] == st[c]["iterations"] == cases[c][1]["iterations"] == 20
        assert math.isclose(st2[c]["final_rel_residual"], cases[c][1]["final_rel_residual"], rel_tol=0)
