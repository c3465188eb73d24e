"""The bias gradient's two kernels: which one a size takes (a tensor shifted by one
element always takes the block per channel, so equal bits mean the same kernel), and
the cluster kernel's sums, exact on small integers, at four to sixteen blocks and
remainders of a block."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _bias(lib, torch, dy, total, cout):
    db = torch.full((cout,), float("nan"), device="cuda")
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.fp_nn_bias_grad(C.c_void_p(dy.data_ptr()), total, cout, C.c_void_p(db.data_ptr()), s) == 0
    return db


@pytest.mark.parametrize("total,cout,block", [(64, 64, True), (4096, 256, True), (12288, 64, True), (24576, 16, True),
                                              (12289, 64, False), (24577, 16, False), (4096, 512, False)])
def test_few_rows_take_a_block_per_channel(gpu_lib, total, cout, block):
    import torch

    g = torch.Generator(device="cuda").manual_seed(total + cout)
    dy = torch.randn(total * cout, generator=g, device="cuda").to(torch.bfloat16)
    shifted = torch.empty(total * cout + 1, dtype=torch.bfloat16, device="cuda")[1:]
    shifted.copy_(dy)
    a, b = _bias(gpu_lib, torch, dy, total, cout), _bias(gpu_lib, torch, shifted, total, cout)
    assert torch.equal(a, b) == block
    d = dy.double().view(total, cout)
    # additions in a row: total / 256 and eight in the block per channel; in the cluster fewer
    # per thread (four blocks of 1024 or more), at most ten in a block and sixteen over the blocks
    bound = (total / 256 + 8 + 10 + 16) * 2.0 ** -24 * d.abs().sum(0)
    for db in (a, b):
        assert bool(((db.double() - d.sum(0)).abs() <= bound).all())


@pytest.mark.parametrize("total,cout", [(24577, 8), (24600, 16), (30001, 32), (70001, 64), (131072, 64), (262147, 8),
                                        (20000, 128), (9001, 512), (5001, 1024)])
def test_cluster_sums_are_exact_on_integers(gpu_lib, total, cout):
    import torch

    g = torch.Generator(device="cuda").manual_seed(total)
    dy = torch.randint(-8, 9, (total, cout), generator=g, device="cuda")  # every partial sum below 2^24
    db = _bias(gpu_lib, torch, dy.to(torch.bfloat16), total, cout)
    assert torch.equal(db.long(), dy.sum(0)) and torch.equal(db, db.round())
