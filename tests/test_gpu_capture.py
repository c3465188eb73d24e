"""Entry points that only queue work on a stream, under a caller's stream capture
and on the default stream: the operator apply (specialised and generic passes), the
allocation-free Green apply, and a convolution layer's four calls, replayed against
the direct calls bit for bit."""
import ctypes as C

import numpy as np
import pytest

from fft_method_test_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


def _replay(torch, stream, call, outs):
    """The results of a captured and replayed call."""
    for o in outs:
        o.zero_()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
        call()
    assert all(not bool(o.any()) for o in outs)  # recorded, not run
    g.replay()
    torch.cuda.synchronize()
    return [o.clone() for o in outs]


@pytest.mark.parametrize("shape,precision", [((32, 32, 32), "mixed"), ((24, 45, 36), "fp64"), ((16, 18, 20), "mixed")])
def test_operator_apply(gpu_lib, shape, precision):
    import torch

    from fft_method_test_gb300.permeability import PermeabilityProblem

    with PermeabilityProblem(shape, precision=precision) as p:
        nb = p.set_geometry(G.gaussian_field(shape, 3.0, 0.45, seed=2))
        x = torch.randn(3 * nb, dtype=torch.float64, device="cuda")
        y = torch.zeros_like(x)
        torch.cuda.synchronize()
        s = torch.cuda.ExternalStream(gpu_lib.fp_stream(p.handle))

        def call():
            assert gpu_lib.fp_operator_apply_device(p.handle, _p(x), _p(y)) == 0

        call()
        torch.cuda.synchronize()
        direct = y.clone()
        assert np.isfinite(direct.cpu().numpy()).all()
        assert torch.equal(_replay(torch, s, call, [y])[0], direct)


def test_green_apply_noalloc(gpu_lib):
    import torch

    n = 24
    f = torch.randn((3, n, n, n), dtype=torch.float64, device="cuda")
    v = torch.zeros_like(f)
    s = torch.cuda.Stream()

    def call(stream):
        assert gpu_lib.fp_green_apply_noalloc(n, n, n, 1.0, 1.0, 2, _p(f), _p(v), C.c_void_p(stream)) == 0

    torch.cuda.synchronize()
    call(0)  # the default stream
    torch.cuda.synchronize()
    direct = v.clone()
    assert bool(direct.any())
    assert torch.equal(_replay(torch, s, lambda: call(s.cuda_stream), [v])[0], direct)


@pytest.mark.parametrize("cin,cout,e,samples", [(16, 32, 16, 2), (64, 128, 4, 4), (128, 64, 16, 4)])
def test_convolution_layer(gpu_lib, cin, cout, e, samples):
    import torch

    total = samples * e ** 3
    bf = lambda *n: torch.randn(n, device="cuda").to(torch.bfloat16)  # noqa: E731
    x, dy, w, b = bf(total, cin), bf(total, cout), bf(27, cout, cin), torch.randn(cout, device="cuda")
    wt = w.transpose(1, 2).contiguous()
    y = torch.zeros((total, cout), dtype=torch.bfloat16, device="cuda")
    dx, dw = torch.zeros((total, cin), device="cuda"), torch.zeros((27, cout, cin), device="cuda")
    db, part = torch.zeros(cout, device="cuda"), torch.empty(-(-total // 1024) * 27 * cout * cin, device="cuda")
    s = torch.cuda.Stream()
    st = C.c_void_p(s.cuda_stream)

    def call():
        wgrad = gpu_lib.fp_nn_wgrad if max(cin, cout) < 128 else gpu_lib.fp_nn_wgrad_cc
        rc = gpu_lib.fp_nn_conv_tc(e, e, e, total, 1, 1, _p(x), cin, _p(w), _p(b), cout, 1, None, _p(y), st)
        rc = rc or gpu_lib.fp_nn_conv_tc(e, e, e, total, 1, -1, _p(dy), cout, _p(wt), None, cin, 0, _p(dx), None, st)
        rc = rc or wgrad(e, e, e, total, 1, _p(dy), cout, _p(x), cin, 1024, _p(part), _p(dw), st)
        assert (rc or gpu_lib.fp_nn_bias_grad(_p(dy), total, cout, _p(db), st)) == 0

    torch.cuda.synchronize()
    outs = [y, dx, dw, db]
    call()
    torch.cuda.synchronize()
    direct = [o.clone() for o in outs]
    captured = _replay(torch, s, call, outs)
    assert all(torch.equal(a, d) and bool(d.any()) for a, d in zip(captured, direct))
