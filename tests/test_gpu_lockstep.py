"""fp_solve_permeability's lockstep of small cells against its load cases solved
one at a time: the same K to the bit and the same iteration counts."""
import numpy as np
import pytest

from fft_method_test_gb300 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,precision,tol", [((32, 32, 32), "fp64", 1e-10), ((20, 45, 24), "fp64", 1e-9),
                                                 ((48, 48, 48), "mixed", 1e-7), ((30, 64, 27), "mixed", 1e-7),
                                                 ((16, 16, 16), "fp64", 1e-10)])
def test_lockstep_equals_single_load_cases(gpu_lib, shape, precision, tol):
    from fft_method_test_gb300.permeability import PermeabilityProblem

    mask = G.gaussian_field(shape, 3.0, 0.45, seed=31)
    with PermeabilityProblem(shape, precision=precision) as p:
        p.set_geometry(mask)
        K, st = p.solve_permeability(tol, 20000)
        K2, _ = p.solve_permeability(tol, 20000)
        assert np.array_equal(K, K2)
        for col in range(3):
            avg, s1, _ = p.solve_load_case(np.eye(3)[col], tol, 20000)
            assert np.array_equal(K[:, col], p.mu * avg)
            assert st[col]["iterations"] == s1["iterations"] and st[col]["converged"] == s1["converged"]


def test_lockstep_reports_errors(gpu_lib):
    from fft_method_test_gb300.permeability import PermeabilityProblem

    with PermeabilityProblem((32, 32, 32)) as p:
        with pytest.raises(Exception):
            p.solve_permeability(1e-8, 100)  # no geometry
        p.set_geometry(G.spheres(32, 4.0, 0.6, seed=12))
        with pytest.raises(ValueError):
            p.solve_permeability(0.0, 100)
        K, st = p.solve_permeability(1e-8, 5)  # stops at the iteration limit
        assert [s["iterations"] for s in st] == [5, 5, 5] and not any(s["converged"] for s in st)
