"""fp_nn_conv_tc's tile form (dilation 1, up to 64 input channels: planes of less
and more than a tile, edges of one voxel, several samples, both signs) and its
per-tap form, the latter on grids large enough for all output channels in one CTA and
small enough to split them (the launch rule of learned_tc.cu), with three and
four buffers, against a float64 convolution."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 64), (64, 32), (64, 128), (128, 64), (128, 128), (112, 64)])
@pytest.mark.parametrize("shape,samples,dil,sign", [((32, 32, 40), 1, 1, 1), ((20, 16, 33), 4, 2, -1), ((9, 5, 3), 1, 1, 1),
                                                     ((20, 16, 33), 2, 1, -1), ((1, 7, 2), 3, 1, -1), ((3, 1, 1), 2, 1, 1),
                                                     ((6, 4, 130), 1, 1, 1)])
def test_conv_tiles(gpu_lib, cin, cout, shape, samples, dil, sign):
    import torch

    nz, ny, nx = shape
    total = samples * nz * ny * nx
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    x = torch.randn((total, cin), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((27, cout, cin), generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    b = torch.randn(cout, generator=g, device="cuda")
    y32 = torch.empty((total, cout), device="cuda")
    y16 = torch.empty((total, cout), dtype=torch.bfloat16, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert gpu_lib.fp_nn_conv_tc(nx, ny, nz, total, dil, sign, p(x), cin, p(w), p(b), cout, 1, p(y32), p(y16), s) == 0
    xs = x.double().view(samples, nz, ny, nx, cin)
    ref = torch.zeros((total, cout), dtype=torch.float64, device="cuda") + b.double()
    for tap in range(27):
        off = [-sign * dil * (tap // 9 - 1), -sign * dil * (tap // 3 % 3 - 1), -sign * dil * (tap % 3 - 1)]
        ref += torch.roll(xs, off, (1, 2, 3)).reshape(total, cin) @ w[tap].double().T
    ref = ref.relu()
    flag = C.c_int(1)
    assert gpu_lib.fp_nn_tc_error(C.byref(flag), 0) == 0 and flag.value == 0
    scale = float(ref.abs().max())
    # FP32 accumulation of 27 cin products
    assert float((y32.double() - ref).abs().max()) < 1e-5 * scale
    assert torch.equal(y16, y32.to(torch.bfloat16))
