"""Weight and bias gradients of one convolution against float64 sums: channel
blocks of 16, 32 and 64 (three taps per block and one), chunks that end inside a
16-voxel step, cells narrower than a step, both entry points, and the calls that
keep the former kernels (unaligned tensors, output counts off the blocks)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


def _case(torch, shape, samples, cin, cout, shift):
    g = torch.Generator(device="cuda").manual_seed(cin * 1000 + cout)
    total = samples * int(np.prod(shape))

    def draw(c):  # `shift` elements into its buffer: 0 keeps 16-byte alignment
        return torch.randn(total * c + 8, generator=g, device="cuda").to(torch.bfloat16)[shift:shift + total * c].view(total, c)

    return total, draw(cin), draw(cout)


def _reference(torch, x, dy, shape, samples, dil):
    xs = x.double().view(samples, *shape, -1)
    d = dy.double()
    out = []
    for tap in range(27):
        off = [dil * (tap // 9 - 1), dil * (tap // 3 % 3 - 1), dil * (tap % 3 - 1)]
        out.append(d.T @ torch.roll(xs, [-o for o in off], (1, 2, 3)).reshape(x.shape))
    return torch.stack(out)


@pytest.mark.parametrize("cin,cout,entry", [(16, 16, "tc"), (32, 16, "tc"), (16, 32, "tc"), (32, 32, "tc"),
                                            (32, 64, "tc"), (64, 32, "tc"), (64, 64, "tc"), (16, 64, "cc"),
                                            (64, 16, "cc"), (48, 80, "cc"), (128, 64, "cc"), (128, 128, "cc")])
@pytest.mark.parametrize("shape,samples,dil,chunk,shift", [((8, 8, 8), 3, 1, 4096, 0), ((4, 6, 10), 2, 2, 1024, 0),
                                                           ((5, 3, 2), 7, 1, 48, 0), ((4, 4, 4), 2, 1, 64, 4)])
def test_weight_gradient(gpu_lib, cin, cout, entry, shape, samples, dil, chunk, shift):
    import torch

    total, x, dy = _case(torch, shape, samples, cin, cout, shift)
    nz, ny, nx = shape
    nchunks = -(-total // chunk)
    partial = torch.full((nchunks * 27 * cout * cin,), float("nan"), device="cuda")
    dw = torch.full((27, cout, cin), float("nan"), device="cuda")
    fn = gpu_lib.fp_nn_wgrad if entry == "tc" else gpu_lib.fp_nn_wgrad_cc
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert fn(nx, ny, nz, total, dil, _p(dy), cout, _p(x), cin, chunk, _p(partial), _p(dw), s) == 0
    ref = _reference(torch, x, dy, shape, samples, dil)
    # FP32 sums of `total` products: total * 2^-24 relative to the sum of magnitudes at most
    scale = (dy.double().abs().T @ x.double().abs()).max()
    assert float((dw.double() - ref).abs().max()) <= max(total, 64) * 2.0 ** -24 * float(scale)


@pytest.mark.parametrize("total,cout,shift", [(1, 8, 0), (7, 16, 0), (5000, 32, 0), (70001, 64, 0), (3000, 128, 0),
                                              (1000, 24, 0), (1000, 5, 0), (1000, 16, 1)])
def test_bias_gradient(gpu_lib, total, cout, shift):
    import torch

    g = torch.Generator(device="cuda").manual_seed(total)
    dy = torch.randn(total * cout + 8, generator=g, device="cuda").to(torch.bfloat16)[shift:shift + total * cout]
    db = torch.full((cout,), float("nan"), device="cuda")
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert gpu_lib.fp_nn_bias_grad(_p(dy), total, cout, _p(db), s) == 0
    d = dy.double().view(total, cout)
    bound = max(total, 64) * 2.0 ** -24 * float(d.abs().sum(0).max())
    assert float((db.double() - d.sum(0)).abs().max()) <= bound
