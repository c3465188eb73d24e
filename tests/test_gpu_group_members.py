"""Lockstep groups against load cases solved one at a time on each member's own
handle (solve_load_case, which never runs the group kernels): members that finish
first, last and in the middle, and a group larger than the active list of the
shared z pass (64 members)."""
import numpy as np
import pytest

from fft_method_test_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _one_by_one(p, tol, maxit):
    K, its = np.zeros((3, 3)), []
    for c in range(3):
        avg, st, _ = p.solve_load_case(np.eye(3)[c], tol, maxit)
        K[:, c] = p.mu * avg
        its.append(st["iterations"])
    return K, its


def _check(masks, precision, tol, maxit=4000):
    from fft_method_test_gb300.permeability import PermeabilityProblem, group_solve_permeability

    ps = []
    try:
        for m in masks:
            ps.append(PermeabilityProblem(m.shape, precision=precision))
            ps[-1].set_geometry(m)
        Kg, stg = group_solve_permeability(ps, tol, maxit)
        totals = []
        for i, p in enumerate(ps):
            K, its = _one_by_one(p, tol, maxit)
            assert np.array_equal(Kg[i], K), i
            assert [s["iterations"] for s in stg[i]] == its, i
            totals.append(sum(its))
        return totals
    finally:
        for p in ps:
            p.close()


@pytest.mark.parametrize("order", [(0, 1, 2), (1, 2, 0), (2, 1, 0)])
@pytest.mark.parametrize("shape,precision,tol", [((32, 32, 32), "fp64", 1e-9), ((48, 30, 64), "mixed", 1e-7)])
def test_members_finish_in_any_order(gpu_lib, order, shape, precision, tol):
    dense = G.gaussian_field(shape, 2.0, 0.35, seed=4)   # many iterations
    middle = G.gaussian_field(shape, 4.0, 0.5, seed=5)
    easy = np.ones(shape, dtype=np.uint8)                # a single post
    easy[:, 4:7, 5:9] = 0
    cells = (easy, middle, dense)
    totals = _check([cells[k] for k in order], precision, tol)
    assert len(set(totals)) == 3 and np.argsort(totals).tolist() == np.argsort(order).tolist()


def test_group_larger_than_the_active_list(gpu_lib):
    _check([G.gaussian_field(20, 2.5, 0.35 + 0.004 * i, seed=100 + i) for i in range(66)], "fp64", 1e-6)
