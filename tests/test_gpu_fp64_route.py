"""FP64 applies of grids whose specialised passes are the slower ones take the
generic passes (bit for bit), next to grids that keep the specialised ones; the
solves on them run one case at a time, with the same results."""
import os

import numpy as np
import pytest

from conftest import rel_err
from fft_method_test_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _apply(shape, precision, off):
    from fft_method_test_gb300.permeability import PermeabilityProblem

    os.environ["FFTPERM_NO_FAST"] = off
    try:
        with PermeabilityProblem(shape, precision=precision) as p:
            nb = p.set_geometry(G.gaussian_field(shape, 3.0, 0.4, seed=162))
            y = p.operator_apply(np.random.default_rng(3).uniform(-1, 1, 3 * nb))
            return y, p.solve_permeability(1e-3, 12)
    finally:
        os.environ.pop("FFTPERM_NO_FAST", None)


# shapes are (nz, ny, nx)
@pytest.mark.parametrize("shape,generic", [((162, 162, 20), True), ((162, 216, 20), True), ((216, 162, 20), False),
                                           ((162, 20, 162), False), ((20, 162, 162), False)])
def test_fp64_route(gpu_lib, shape, generic):
    y, (K, st) = _apply(shape, "fp64", "0")
    y0, (K0, st0) = _apply(shape, "fp64", "1")
    assert np.array_equal(y, y0) == generic and rel_err(y, y0) < 1e-13
    assert np.array_equal(K, K0) == generic and rel_err(K, K0) < 1e-9
    assert [s["iterations"] for s in st] == [s["iterations"] for s in st0]


def test_mixed_precision_keeps_the_specialised_passes(gpu_lib):
    y, _ = _apply((162, 162, 20), "mixed", "0")
    y0, _ = _apply((162, 162, 20), "mixed", "1")
    assert not np.array_equal(y, y0) and rel_err(y, y0) < 2e-6
