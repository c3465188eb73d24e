"""Brinkman iteration where br_div hands over to the division.

The two-operation quotient holds for 2^-600 <= |x| < 2^600 (about 2.4e-181 to
4.1e180); smaller and larger dividends, subnormals, infinities and NaN divide.
The kernels follow the oracle expression by expression, so finite fields agree
to 1e-14 of their largest value, or within a few of the smallest subnormals."""
import numpy as np
import pytest

from fft_method_test_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def cell():
    return G.to_ids((np.random.default_rng(21).random((9, 6, 33)) >= 0.4).astype(np.uint8))


@pytest.mark.parametrize("force", [(1e-200, -1e-190, 0.0), (1e-170, 0.0, 1e-185), (0.0, 3e-181, 2e-181),
                                   (1e-310, 0.0, 2e-312), (0.0, 1e-320, 0.0), (1e150, 0.0, 1e140)])
def test_tiny_and_large_forces_match_oracle(gpu_lib, restatement, force):
    from fft_method_test_gb300.permeability import solveBrinkman

    ids = cell()
    ro = restatement.brinkman(ids, 1, 1.0, 1e4, 0.9, 1e-8, 12, force, want_fields=True)
    r = solveBrinkman(ids, force, fluid_mu=1.0, solid_penalty=1e4, max_iterations=12, want_fields=True)
    assert r["iterations"] == ro["iterations"]
    for f in ("ux", "uy", "uz", "p"):
        bound = 1e-14 * np.abs(ro[f]).max() + 8 * 5e-324
        assert np.abs(r[f].ravel() - ro[f]).max() <= bound, f


@pytest.mark.parametrize("force", [(1e200, 0.0, 0.0), (np.inf, 0.0, 0.0), (0.0, -np.inf, 1.0),
                                   (0.0, 0.0, np.nan)])
def test_overflow_infinities_and_nan_are_reported(gpu_lib, restatement, force):
    from fft_method_test_gb300._capi import FpError
    from fft_method_test_gb300.permeability import solveBrinkman

    ids = cell()
    with pytest.raises(RuntimeError):
        restatement.brinkman(ids, 1, 1.0, 1e4, 0.9, 1e-8, 12, force)
    with pytest.raises(FpError) as ei:
        solveBrinkman(ids, force, fluid_mu=1.0, solid_penalty=1e4, max_iterations=12)
    assert "unstable" in str(ei.value)
