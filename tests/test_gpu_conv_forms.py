"""Every form of fp_nn_conv_tc that the rule can choose (tile form and per-tap form,
16 to 128 output channels per CTA, two to four buffers) against a float64
convolution, at sizes whose choice test_conv_rules_cpu.py checks."""
import ctypes as C

import pytest

from test_conv_rules_cpu import FORMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("sign", [1, -1])
def test_conv_form(gpu_lib, form, sign):
    import torch

    nx, ny, nz, samples, cin, cout, dil = FORMS[form]
    total = samples * nz * ny * nx
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    x = torch.randn((total, cin), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((27, cout, cin), generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    b = torch.randn(cout, generator=g, device="cuda")
    y32 = torch.full((total, cout), float("nan"), device="cuda")
    y16 = torch.full((total, cout), float("nan"), dtype=torch.bfloat16, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert gpu_lib.fp_nn_conv_tc(nx, ny, nz, total, dil, sign, p(x), cin, p(w), p(b), cout, 1, p(y32), p(y16), s) == 0
    xs = x.double().view(samples, nz, ny, nx, cin)
    ref = torch.zeros((total, cout), dtype=torch.float64, device="cuda") + b.double()
    mag = ref.abs()
    for tap in range(27):
        off = [-sign * dil * (tap // 9 - 1), -sign * dil * (tap // 3 % 3 - 1), -sign * dil * (tap % 3 - 1)]
        xt = torch.roll(xs, off, (1, 2, 3)).reshape(total, cin)
        ref += xt @ w[tap].double().T
        mag += xt.abs() @ w[tap].double().abs().T
    flag = C.c_int(1)
    assert gpu_lib.fp_nn_tc_error(C.byref(flag), 0) == 0 and flag.value == 0
    # FP32 sums of 27 cin products and the bias: each addition rounds by 2^-24 of a partial sum
    bound = (27 * cin + 1) * 2.0 ** -24 * mag
    assert bool(((y32.double() - ref.relu()).abs() <= bound).all())
    assert torch.equal(y16, y32.to(torch.bfloat16))
