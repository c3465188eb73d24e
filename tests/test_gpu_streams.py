"""Solves beside other work of the same process: a solve returns while another
stream's kernel still runs (nothing in it waits for the whole device), and threads
that solve at once get what each gets alone."""
import threading

import numpy as np
import pytest

from fft_method_test_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _problem(n, precision, seed):
    from fft_method_test_gb300.permeability import PermeabilityProblem

    mask = G.gaussian_field(n, 3.0, 0.45, seed=seed)
    p = PermeabilityProblem(mask.shape, precision=precision)
    p.set_geometry(mask)
    return p


@pytest.mark.parametrize("how", ["permeability", "block", "group"])
def test_solve_does_not_wait_for_other_streams(gpu_lib, how):
    import torch

    from fft_method_test_gb300.permeability import group_solve_permeability

    ps = [_problem(32, "mixed", s) for s in (1, 2)]

    def solve():
        if how == "group":
            return group_solve_permeability(ps, 1e-5)[0]
        return ps[0].solve_permeability(1e-5, 2000, block=how == "block")[0]

    try:
        K = solve()  # modules, memory pool and pinned blocks
        other, done = torch.cuda.Stream(), torch.cuda.Event()
        with torch.cuda.stream(other):
            torch.cuda._sleep(int(2e9))  # about a second of one thread's clock
            done.record()
        K2 = solve()
        assert not done.query(), "the solve waited for another stream's kernel"
        done.synchronize()
        assert np.array_equal(K, K2)
    finally:
        for p in ps:
            p.close()


def test_threads_solve_at_once(gpu_lib):
    ps = [_problem(32, "mixed", 4), _problem(48, "mixed", 5), _problem(32, "fp64", 6)]
    try:
        alone = [p.solve_permeability(1e-6, 4000)[0] for p in ps]
        got = [None] * len(ps)

        def work(i):
            got[i] = [ps[i].solve_permeability(1e-6, 4000)[0] for _ in range(3)]

        threads = [threading.Thread(target=work, args=(i,)) for i in range(len(ps))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for i, K in enumerate(alone):
            assert all(np.array_equal(K, k) for k in got[i]), i
    finally:
        for p in ps:
            p.close()
