"""The block and group solves against load cases solved one at a time
(solve_load_case runs neither): grids with specialised passes, and grids without,
where the block and the group fall back to the members' single solves."""
import os
import re

import numpy as np
import pytest

from conftest import ROOT
from fft_method_test_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _specialised(n):
    src = open(os.path.join(ROOT, "fft_method_test_gb300", "csrc", "fft_fast.cuh")).read()
    src = src[src.index("#define FP_FAST_EDGES"):]
    return n in {int(v) for v in re.findall(r"CALL\((\d+)\)", src[:src.index("\n\n")])}


def _one_by_one(p, tol, maxit=20000):
    K, its = np.zeros((3, 3)), []
    for c in range(3):
        avg, st, _ = p.solve_load_case(np.eye(3)[c], tol, maxit)
        K[:, c] = p.mu * avg
        its.append(st["iterations"])
    return K, its


@pytest.mark.parametrize("shape,precision,tol,specialised", [
    ((32, 32, 32), "fp64", 1e-10, True), ((48, 48, 48), "mixed", 1e-7, True), ((64, 64, 64), "mixed", 1e-7, True),
    ((27, 36, 45), "fp64", 1e-9, True), ((16, 16, 16), "fp64", 1e-10, False), ((18, 32, 24), "mixed", 1e-7, False),
    ((32, 18, 32), "fp64", 1e-9, False), ((20, 20, 125), "mixed", 1e-7, False)])
def test_block_and_group_equal_load_cases(gpu_lib, shape, precision, tol, specialised):
    from fft_method_test_gb300.permeability import PermeabilityProblem, group_solve_permeability

    assert all(map(_specialised, shape)) == specialised
    ps = []
    try:
        for seed in (7, 8):
            ps.append(PermeabilityProblem(shape, precision=precision))
            ps[-1].set_geometry(G.gaussian_field(shape, 3.0, 0.42, seed=seed))
        Kg, stg = group_solve_permeability(ps, tol)
        for i, p in enumerate(ps):
            K, its = _one_by_one(p, tol)
            Kb, stb = p.solve_permeability(tol, 20000, block=True)
            Kp, stp = p.solve_permeability(tol, 20000)
            for other, st in ((Kg[i], stg[i]), (Kb, stb), (Kp, stp)):
                assert np.array_equal(K, other)
                assert [s["iterations"] for s in st] == its
                assert all(s["converged"] for s in st)
    finally:
        for p in ps:
            p.close()
