"""fp_set_tiling's cap on the x rows of a CTA: any value is accepted and none asks
for more threads than the specialised x passes hold (240 and 256 take 16 threads
per line, 225 eight, 160 four), against the generic passes."""
import numpy as np
import pytest

from conftest import rel_err
from fft_method_test_gb300 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [240, 256, 225, 160])
@pytest.mark.parametrize("precision,bar", [("fp64", 1e-13), ("mixed", 2e-6)])
def test_any_x_rows_cap(gpu_lib, nx, precision, bar):
    from fft_method_test_gb300.permeability import PermeabilityProblem

    shape = (20, 24, nx)
    with PermeabilityProblem(shape, precision=precision) as p:
        nb = p.set_geometry(G.gaussian_field(shape, 3.0, 0.4, seed=nx))
        x = np.random.default_rng(nx).uniform(-1, 1, 3 * nb)
        p.set_tiling(tma=False)
        ref = p.operator_apply(x)
        for rows in (2, 3, 16, 17, 18, 24, 32, 1000):
            p.set_tiling(x_rows=rows)
            assert rel_err(p.operator_apply(x), ref) < bar, rows
