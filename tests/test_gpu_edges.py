"""The specialised passes of the edges in fft_edges.cuh against the generic
passes, each edge along x, y and z (tile remainders, odd edges, idle owners),
and a group solve of such a grid against its single solves."""
import os
import re

import numpy as np
import pytest

from conftest import ROOT, rel_err
from fft_method_test_gb300 import geometry as G

pytestmark = pytest.mark.gpu

EDGES = [int(n) for n in re.findall(r"\bE\((\d+),", open(
    os.path.join(ROOT, "fft_method_test_gb300", "csrc", "fft_edges.cuh")).read())]


def _applies(shape, precision, mask, x, off):
    from fft_method_test_gb300.permeability import PermeabilityProblem

    os.environ["FFTPERM_NO_FAST"] = off
    try:
        with PermeabilityProblem(shape, precision=precision) as p:
            nb = p.set_geometry(mask)
            v = np.random.default_rng(2).uniform(-1, 1, 3 * nb) if x is None else x
            outs = [v, p.operator_apply(v)]
            p.set_tiling(lowreg=True, x_rows=2)  # single-stage z pass, short x tiles
            outs.append(p.operator_apply(v))
            return outs
    finally:
        os.environ.pop("FFTPERM_NO_FAST", None)


@pytest.mark.parametrize("n", EDGES)
@pytest.mark.parametrize("precision,bar", [("fp64", 1e-13), ("mixed", 2e-6)])
def test_edge_matches_generic_passes(gpu_lib, n, precision, bar):
    for shape in ((20, 27, n), (24, n, 30), (n, 25, 20)):
        mask = G.gaussian_field(shape, 3.0, 0.4, seed=n)
        x, y0, _ = _applies(shape, precision, mask, None, "1")
        _, y1, y2 = _applies(shape, precision, mask, x, "0")
        assert rel_err(y1, y0) < bar, shape
        assert rel_err(y2, y0) < bar, shape


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-7)])
def test_group_of_uneven_edges_equals_single_solves(gpu_lib, precision, tol):
    from fft_method_test_gb300.permeability import PermeabilityProblem, group_solve_permeability

    masks = [G.gaussian_field((45, 36, 27), 3.0, 0.4, seed=s) for s in (1, 2, 3)]
    ps = []
    try:
        for m in masks:
            p = PermeabilityProblem(m.shape, precision=precision)
            ps.append(p)
            p.set_geometry(m)
        Kg, _ = group_solve_permeability(ps, tol)
        for p, K in zip(ps, Kg):
            assert np.array_equal(K, p.solve_permeability(tol, 20000)[0])
    finally:
        for p in ps:
            p.close()
