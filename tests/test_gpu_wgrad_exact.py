"""The weight gradient on small integers, whose FP32 sums are exact, so that a
lost row, tap, chunk or warp cannot pass: both kernels and both entry points, chunks
that end inside a step; and which kernel a chunk takes (tensors shifted by one
element always take the former one, so equal bits mean the same kernel)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _wgrad(lib, torch, entry, shape, x, dy, dil, chunk):
    total, cin = x.shape
    cout = dy.shape[1]
    nz, ny, nx = shape
    part = torch.full((-(-total // chunk) * 27 * cout * cin,), float("nan"), device="cuda")
    dw = torch.full((27, cout, cin), float("nan"), device="cuda")
    fn = lib.fp_nn_wgrad if entry == "tc" else lib.fp_nn_wgrad_cc
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert fn(nx, ny, nz, total, dil, p(dy), cout, p(x), cin, chunk, p(part), p(dw), s) == 0
    return dw


def _shifted(torch, t):
    out = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("cin,cout,entry", [(16, 16, "tc"), (16, 32, "tc"), (32, 32, "tc"), (64, 32, "tc"),
                                            (64, 64, "tc"), (64, 16, "cc"), (48, 80, "cc"), (128, 128, "cc")])
@pytest.mark.parametrize("shape,samples,dil,chunk", [((8, 8, 8), 3, 1, 4096), ((12, 9, 7), 5, 2, 1024),
                                                     ((5, 3, 2), 30, 1, 112), ((6, 6, 6), 4, 1, 48)])
def test_exact_on_integers(gpu_lib, cin, cout, entry, shape, samples, dil, chunk):
    import torch

    total = samples * int(np.prod(shape))
    g = torch.Generator(device="cuda").manual_seed(cin + cout + total)
    x = torch.randint(-8, 9, (total, cin), generator=g, device="cuda")  # sums below 64 * 4000 < 2^24
    dy = torch.randint(-8, 9, (total, cout), generator=g, device="cuda")
    dw = _wgrad(gpu_lib, torch, entry, shape, x.to(torch.bfloat16), dy.to(torch.bfloat16), dil, chunk)
    xs = x.double().view(samples, *shape, cin)
    for tap in range(27):
        off = [-dil * (tap // 9 - 1), -dil * (tap // 3 % 3 - 1), -dil * (tap % 3 - 1)]
        ref = dy.double().T @ torch.roll(xs, off, (1, 2, 3)).reshape(total, cin)
        assert torch.equal(dw[tap].double(), ref), tap


@pytest.mark.parametrize("cin,cout,chunk,former", [(64, 64, 176, True), (64, 64, 192, False), (64, 32, 112, True),
                                                   (64, 32, 128, False), (32, 32, 48, True), (32, 32, 64, False),
                                                   (16, 16, 16, False)])
def test_short_chunks_keep_the_former_kernel(gpu_lib, cin, cout, chunk, former):
    import torch

    shape, total = (10, 9, 8), 4 * 720
    g = torch.Generator(device="cuda").manual_seed(chunk)
    x = torch.randn((total, cin), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn((total, cout), generator=g, device="cuda").to(torch.bfloat16)
    a = _wgrad(gpu_lib, torch, "tc", shape, x, dy, 1, chunk)
    b = _wgrad(gpu_lib, torch, "tc", shape, _shifted(torch, x), _shifted(torch, dy), 1, chunk)
    assert torch.equal(a, b) == former
