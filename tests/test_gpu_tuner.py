"""What the autotuner times is what an iteration runs: the launches of an apply in
fp_time_apply against those of a MINRES iteration without its two vector kernels,
for the specialised passes, the generic ones by tiling, and a generic grid."""
import ctypes as C

import pytest

from fft_method_test_gb300 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,tma", [(32, True), (32, False), (18, True), (18, False)])
def test_timed_apply_is_the_iterations(gpu_lib, monkeypatch, n, tma):
    from fft_method_test_gb300.permeability import PermeabilityProblem

    monkeypatch.setenv("FFTPERM_NO_GRAPHS", "1")
    launches = gpu_lib.fp_kernel_launch_count
    with PermeabilityProblem((n, n, n), precision="fp64") as p:
        p.set_geometry(G.gaussian_field(n, 3.0, 0.45, seed=n))
        p.set_tiling(tma=tma)

        def solve(maxit):
            c0 = launches()
            p.solve_load_case((1.0, 0.0, 0.0), 1e-14, maxit)
            return launches() - c0

        def timed(reps):
            ms = C.c_double()
            c0 = launches()
            assert gpu_lib.fp_time_apply(p.handle, reps, C.byref(ms)) == 0 and ms.value > 0
            return launches() - c0

        iteration = (solve(32) - solve(16)) / 16  # iterations run in chunks of 16
        apply = timed(8) - timed(7)
        assert apply == iteration - 2
