"""What this framework is measured on: the calls a user makes, over the sizes
they are made at.

Kinds of case (every one through a public entry point):

* ``solve``     the permeability tensor of one cell (three load cases), the
                framework's purpose: 32^3 in FP64 (parity with the reference's
                CPU results), 64^3 mixed (an ordinary cell), 256^3 mixed with
                the three load cases as one block (the benchmark cell).
* ``batch``     a queue of uneven microstructures, as an RVE study submits.
* ``apply``     one variational operator apply on device vectors, what a user's
                own Krylov solver calls: small, ragged (edges without
                specialised passes), FP64 and the largest.
* ``flow``      right-hand side and velocity field of a given force (post-
                processing of a solve: full-grid FP64 transforms).
* ``brinkman``  a fixed number of the reference's Brinkman iterations.
* ``fixed``     the Brinkman problem solved to its discrete fixed point.
* ``conv``      one convolution layer of the learned warm start, forward and
                backward, as a training step runs it.

Mixed-precision results carry single-precision accuracy (FP32 transforms and
Green table), so they are kept in float32; FP64 results stay float64.
"""
import ctypes
import math

import numpy as np
import torch

from fft_method_test_gb300 import _capi
from fft_method_test_gb300 import permeability as pm

# grid edges the transforms accept: products of 2, 3 and 5
SMOOTH = sorted(2 ** a * 3 ** b * 5 ** c for a in range(9) for b in range(6) for c in range(4)
                if 8 <= 2 ** a * 3 ** b * 5 ** c <= 256)
# (cin, cout, refinement level below the cell) of the U-Net's convolutions
LAYERS = [(16, 16, 0), (16, 32, 1), (32, 64, 2), (64, 128, 3), (128, 128, 3), (128, 64, 3),
          (64, 32, 2), (32, 16, 1)]


def listed():
    return [
        # smallest whole solve: a parity check against the reference's CPU K
        dict(name="solve_32_fp64", kind="solve", nx=32, ny=32, nz=32, precision="fp64", tol=1e-10,
             phi=0.6, ell=3.0, block=False, tune=False),
        # an ordinary cell with the defaults a first-time user has
        dict(name="solve_64_mixed", kind="solve", nx=64, ny=64, nz=64, precision="mixed", tol=1e-7,
             phi=0.45, ell=5.0, block=False, tune=False),
        # the benchmark cell (Gaussian random field, porosity 0.35), tuned and as a block
        dict(name="solve_256_mixed_block", kind="solve", nx=256, ny=256, nz=256, precision="mixed",
             tol=1e-7, phi=0.35, ell=6.0, block=True, tune=True),
        # an RVE study: uneven cells solved together
        dict(name="batch_uneven_mixed", kind="batch", edges="48,48,48,64,64,64,80,80,96,96",
             precision="mixed", tol=1e-7, max_group=16),
        # operator applies on device vectors
        dict(name="apply_48_mixed", kind="apply", nx=48, ny=48, nz=48, precision="mixed", phi=0.4),
        dict(name="apply_ragged_mixed", kind="apply", nx=100, ny=90, nz=72, precision="mixed",
             phi=0.4),
        dict(name="apply_128_fp64", kind="apply", nx=128, ny=128, nz=128, precision="fp64", phi=0.4),
        dict(name="apply_256_mixed", kind="apply", nx=256, ny=256, nz=256, precision="mixed",
             phi=0.35),
        # right-hand side and velocity field of a load case
        dict(name="flow_96_fp64", kind="flow", nx=96, ny=96, nz=96, phi=0.4),
        # the reference's Brinkman iteration on spheres of radius 8 (128^3, the size it is
        # compared with the variational tensor at)
        dict(name="brinkman_128", kind="brinkman", nx=128, ny=128, nz=128, phi=0.45, iterations=40),
        # its fixed point
        dict(name="fixed_point_48", kind="fixed", nx=48, ny=48, nz=48, phi=0.45, tol=1e-8),
        # a U-Net layer of a training step on four 64^3 cells
        dict(name="conv_16_32_level1", kind="conv", edge=32, samples=4, cin=16, cout=32),
    ]


def _log(rng, lo, hi):
    """An edge of SMOOTH, uniform in its logarithm over [lo, hi]."""
    e = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((n for n in SMOOTH if lo <= n <= hi), key=lambda n: abs(n - e))


def _dims(rng, lo, hi):
    """Cubic cells for half of the draws, as RVE cells are; three edges of their own otherwise."""
    if rng.random() < 0.5:
        n = _log(rng, lo, hi)
        return dict(nx=n, ny=n, nz=n)
    return dict(nx=_log(rng, lo, hi), ny=_log(rng, lo, hi), nz=_log(rng, lo, hi))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "apply", "apply", "apply", "flow", "brinkman",
                       "fixed", "conv", "conv"])
    phi = round(rng.uniform(0.3, 0.6), 3)
    if kind == "solve":
        precision = rng.choice(["fp64", "mixed", "mixed"])
        dims = _dims(rng, 20, 48) if precision == "fp64" else _dims(rng, 32, 128)
        return dict(kind="solve", precision=precision, tol=1e-10 if precision == "fp64" else 1e-7,
                    phi=phi, ell=round(rng.uniform(3.0, 6.0), 2), block=rng.random() < 0.5, tune=False,
                    **dims)
    if kind == "batch":
        edges = [rng.choice([48, 64, 80, 96]) for _ in range(rng.randint(4, 12))]
        return dict(kind="batch", edges=",".join(map(str, edges)), precision="mixed", tol=1e-7,
                    max_group=rng.choice([4, 16]))
    if kind == "apply":
        precision = rng.choice(["fp64", "mixed", "mixed"])
        return dict(kind="apply", precision=precision, phi=phi,
                    **_dims(rng, 24, 160 if precision == "fp64" else 256))
    if kind == "flow":
        return dict(kind="flow", phi=phi, **_dims(rng, 32, 128))
    if kind == "brinkman":
        return dict(kind="brinkman", phi=phi, iterations=rng.randint(10, 40), **_dims(rng, 32, 128))
    if kind == "fixed":
        return dict(kind="fixed", phi=phi, tol=1e-8, **_dims(rng, 24, 64))
    cin, cout, level = rng.choice(LAYERS)
    return dict(kind="conv", edge=rng.choice([32, 48, 64, 96, 128]) >> level, samples=rng.randint(1, 4),
                cin=cin, cout=cout)


# ---- inputs ------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _field_mask(nx, ny, nz, phi, ell, seed):
    """Thresholded Gaussian random field, (nz, ny, nx), 1 = fluid."""
    noise = torch.randn((nz, ny, nx), generator=_generator(seed), device="cuda", dtype=torch.float32)
    k2 = (torch.fft.fftfreq(nz, device="cuda").square()[:, None, None]
          + torch.fft.fftfreq(ny, device="cuda").square()[None, :, None]
          + torch.fft.rfftfreq(nx, device="cuda").square()[None, None, :])
    f = torch.fft.irfftn(torch.fft.rfftn(noise) * torch.exp(-2.0 * math.pi ** 2 * ell ** 2 * k2),
                         s=(nz, ny, nx))
    cut = torch.sort(f.reshape(-1)).values[int(round(phi * f.numel()))]
    return (f < cut).to(torch.uint8)


def _sphere_mask(nx, ny, nz, phi, radius, seed):
    """Overlapping solid spheres in a periodic cell, 1 = fluid."""
    rng = np.random.default_rng(seed)
    count = max(1, int(round(-math.log(phi) * nx * ny * nz / (4.0 / 3.0 * math.pi * radius ** 3))))
    solid = torch.zeros((nz, ny, nx), dtype=torch.bool, device="cuda")
    for c in rng.uniform(0.0, 1.0, size=(count, 3)):
        d2 = 0
        for axis, (n, u) in enumerate(zip((nz, ny, nx), c)):
            d = torch.arange(n, device="cuda", dtype=torch.float32) + 0.5 - float(u) * n
            d = d - n * torch.round(d / n)
            d2 = d2 + d.square().reshape([-1 if a == axis else 1 for a in range(3)])
        solid |= d2 <= radius * radius
    return (~solid).to(torch.uint8)


def _mask(case, seed):
    dims = case["nx"], case["ny"], case["nz"]
    if case["kind"] in ("apply", "flow"):
        seed = 1003  # the cell a program keeps; the vectors come from the seed
    if case["kind"] in ("brinkman", "fixed"):
        return _sphere_mask(*dims, case["phi"], min(8.0, min(dims) / 6), seed)
    return _field_mask(*dims, case["phi"], case.get("ell", 6.0), seed)


def _batch_masks(case, seed):
    out = []
    for i, e in enumerate(map(int, case["edges"].split(","))):
        phi = 0.35 + 0.4 * ((seed * 7 + i * 5) % 11) / 10
        if i % 2:
            out.append(_sphere_mask(e, e, e, phi, 6.0, seed * 100 + i))
        else:
            out.append(_field_mask(e, e, e, phi, 6.0, seed * 100 + i))
    return out


def _vector(n, seed):
    return torch.randn(n, generator=_generator(seed + 12345), device="cuda", dtype=torch.float64)


def _conv_inputs(case, seed):
    g = _generator(seed)
    total = case["samples"] * case["edge"] ** 3
    cin, cout = case["cin"], case["cout"]
    x = torch.randn((total, cin), generator=g, device="cuda").relu().to(torch.bfloat16)
    dy = torch.randn((total, cout), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn((27, cout, cin), generator=g, device="cuda") * math.sqrt(2.0 / (27 * cin))
    w = w.to(torch.bfloat16)
    b = torch.randn(cout, generator=g, device="cuda")
    return x, dy, w, b


GRAD = (0.36, -0.48, 0.8)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return dict(case=case, masks=[m.cpu().numpy() for m in _batch_masks(case, seed)])
    if kind == "conv":
        x, dy, w, b = _conv_inputs(case, seed)
        total, cin, cout = x.shape[0], case["cin"], case["cout"]
        chunk = 4096 if cin < 128 and cout < 128 else 1024  # as the network's training step chooses
        return dict(case=case, lib=_capi.load(), x=x, dy=dy, w=w, wt=w.transpose(1, 2).contiguous(), b=b,
                    chunk=chunk, y=torch.empty((total, cout), dtype=torch.bfloat16, device="cuda"),
                    dx=torch.empty((total, cin), device="cuda"), dw=torch.empty((27, cout, cin), device="cuda"),
                    db=torch.empty(cout, device="cuda"),
                    partial=torch.empty(-(-total // chunk) * 27 * cout * cin, device="cuda"))
    mask = _mask(case, seed).cpu().numpy()
    if kind in ("brinkman", "fixed"):
        return dict(case=case, ids=np.where(mask != 0, 1, 2).astype(np.uint32))
    prob = pm.PermeabilityProblem(mask.shape, precision=case.get("precision", "fp64"))
    prob.set_geometry(mask)
    state = dict(case=case, prob=prob)
    if case.get("tune"):
        prob.autotune()
    if kind == "apply":
        state["x"] = _vector(3 * prob.nb, seed)
        state["y"] = torch.zeros_like(state["x"])
        if case["precision"] == "mixed":
            state["y32"] = torch.zeros(3 * prob.nb, dtype=torch.float32, device="cuda")
            state["stream"] = torch.cuda.ExternalStream(prob.lib.fp_stream(prob.handle))
        torch.cuda.synchronize()  # the handle's stream is not torch's
    elif kind == "flow":
        state["x"] = _vector(3 * prob.nb, seed).cpu().numpy()
    return state


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        K, _ = state["prob"].solve_permeability(case["tol"], 20000, block=case["block"])
        return K.astype(np.float32) if case["precision"] == "mixed" else K
    if kind == "batch":
        K, _, status = pm.batch_solve_permeability(state["masks"], precision=case["precision"], tol=case["tol"],
                                                   max_group=case["max_group"])
        return [K.astype(np.float32), np.array(status)]
    if kind == "apply":
        prob = state["prob"]
        rc = prob.lib.fp_operator_apply_device(prob.handle, _ptr(state["x"]), _ptr(state["y"]))
        if rc != _capi.FP_OK:
            _capi.check(prob.lib, prob.handle, rc)
        if case["precision"] == "fp64":
            return state["y"]
        with torch.cuda.stream(state["stream"]):
            return state["y32"].copy_(state["y"])
    if kind == "flow":
        b = state["prob"].build_rhs(GRAD)
        avg, v = state["prob"].recover(GRAD, state["x"], want_field=True)
        return [b, avg, v]
    if kind == "brinkman":
        r = pm.solveBrinkman(state["ids"], (1.0, 0.0, 0.0), tolerance=1e-30,
                             max_iterations=case["iterations"], want_fields=True)
        return [r["superficialVelocity"], r["ux"], r["uy"], r["uz"], r["p"], r["iterations"]]
    if kind == "fixed":
        r = pm.solveBrinkmanFixedPoint(state["ids"], (1.0, 0.0, 0.0), tolerance=case["tol"], want_fields=True)
        return [r["superficialVelocity"], r["ux"], r["uy"], r["uz"]]
    # conv: forward (bias, ReLU, BF16 out), data gradient (FP32 out), weight and bias gradients
    lib, e, total = state["lib"], case["edge"], state["x"].shape[0]
    cin, cout, chunk = case["cin"], case["cout"], state["chunk"]
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = lib.fp_nn_conv_tc(e, e, e, total, 1, 1, _ptr(state["x"]), cin, _ptr(state["w"]), _ptr(state["b"]), cout, 1,
                           None, _ptr(state["y"]), s)
    rc = rc or lib.fp_nn_conv_tc(e, e, e, total, 1, -1, _ptr(state["dy"]), cout, _ptr(state["wt"]), None, cin, 0,
                                 _ptr(state["dx"]), None, s)
    wgrad = lib.fp_nn_wgrad if cin < 128 and cout < 128 else lib.fp_nn_wgrad_cc
    rc = rc or wgrad(e, e, e, total, 1, _ptr(state["dy"]), cout, _ptr(state["x"]), cin, chunk, _ptr(state["partial"]),
                     _ptr(state["dw"]), s)
    rc = rc or lib.fp_nn_bias_grad(_ptr(state["dy"]), total, cout, _ptr(state["db"]), s)
    if rc != _capi.FP_OK:
        raise _capi.FpError(rc, "convolution layer")
    return [state["y"], state["dx"], state["dw"], state["db"]]


# ---- the work of a pass --------------------------------------------------------


def _apply_work(n, nh, precision):
    """Compact vector in and out, support indices, Green table; six 1-D FFT
    sweeps of three real fields and the 3x3 Green multiply."""
    g = 4 if precision == "mixed" else 8
    nb = 0.11 * n  # support voxels of the fields above
    return (2 * 24 + 4) * nb + 6 * g * nh, 15.0 * n * math.log2(n) + 36.0 * nh


def work(case):
    kind = case["kind"]
    if kind == "conv":
        total = case["samples"] * case["edge"] ** 3
        cin, cout = case["cin"], case["cout"]
        return dict(bytes=total * (2 * cin + 2 * cout + 2 * cout + 4 * cin) + 27 * cin * cout * 8,
                    flops=3 * 2 * 27.0 * total * cin * cout)
    if kind == "batch":
        w = [work(dict(kind="solve", nx=e, ny=e, nz=e, precision=case["precision"], tol=case["tol"]))
             for e in map(int, case["edges"].split(","))]
        return dict(bytes=sum(x["bytes"] for x in w), flops=sum(x["flops"] for x in w))
    n = case["nx"] * case["ny"] * case["nz"]
    nh = (case["nx"] // 2 + 1) * case["ny"] * case["nz"]
    if kind == "apply":
        b, f = _apply_work(n, nh, case["precision"])
        return dict(bytes=b, flops=f)
    if kind == "solve":
        # nominal iterations per load case (about 900 at 256^3 and 1e-7, growing with the edge);
        # an iteration is an apply and the Lanczos updates (v, v_old, w, w_old, x read; v, w, x written)
        its = 3 * 56 * n ** (1 / 6) * -math.log10(case["tol"]) / 7
        b, f = _apply_work(n, nh, case["precision"])
        return dict(bytes=its * (b + 8 * 24 * 0.11 * n), flops=its * (f + 60 * 0.11 * n))
    if kind == "flow":
        return dict(bytes=1.0 * n + 3 * 8 * n + 3 * 24 * 0.11 * n + 2 * 48 * nh, flops=2 * (15.0 * n * math.log2(n)))
    if kind == "brinkman":
        # ids in, four fields out; 35 pressure sweeps of 7 operations, momentum, divergence, projection
        return dict(bytes=36.0 * n, flops=case["iterations"] * n * (35 * 7.0 + 50))
    # fixed point: nominal CG iterations, two FP64 transforms each
    its = 18 * max(case["nx"], case["ny"], case["nz"])
    return dict(bytes=28.0 * n, flops=its * (2 * 7.5 * n * math.log2(n) + 80 * n))


# ---- the same in 64 bits, by plain torch ----------------------------------------


def _green(nx, ny, nz, p_radius=2):
    """(6, nz, ny, nx/2+1) symmetrised energy-consistent Green tensor (xx xy xz
    yy yz zz), voxel size 1, viscosity 1: real part of what the inverse
    transform of a real field keeps."""
    def at(kx, ky, kz):
        g = torch.zeros((6, kz.numel(), ky.numel(), kx.numel()), dtype=torch.float64, device="cuda")

        def axis(k, n, p, dim):
            m = (k + p * n).double()
            s = torch.where(m == 0, torch.ones_like(m), torch.sin(math.pi * m / n) / (math.pi * m / n))
            s = torch.where((m != 0) & (m.remainder(n) == 0), torch.zeros_like(s), s)
            shape = [1, 1, 1]
            shape[dim] = -1
            return s.square().reshape(shape), (2 * math.pi * m / n).reshape(shape)

        r = range(-p_radius, p_radius + 1)
        for pz in r:
            wz, qz = axis(kz, nz, pz, 0)
            for py in r:
                wy, qy = axis(ky, ny, py, 1)
                for px in r:
                    wx, qx = axis(kx, nx, px, 2)
                    q2 = qx * qx + qy * qy + qz * qz
                    f = torch.where(q2 > 0, wx * wy * wz / q2, torch.zeros_like(q2))
                    f2 = torch.where(q2 > 0, f / q2, torch.zeros_like(q2))
                    g[0] += f - f2 * (qx * qx)
                    g[1] -= f2 * (qx * qy)
                    g[2] -= f2 * (qx * qz)
                    g[3] += f - f2 * (qy * qy)
                    g[4] -= f2 * (qy * qz)
                    g[5] += f - f2 * (qz * qz)
        return g

    kx, ky, kz = (torch.arange(n, device="cuda") for n in (nx // 2 + 1, ny, nz))
    g = 0.5 * (at(kx, ky, kz) + at((-kx) % nx, (-ky) % ny, (-kz) % nz))
    g[:, 0, 0, 0] = 0
    return g


def _support(mask):
    """Solid voxels with a fluid voxel among their 26 periodic neighbours, ascending."""
    near = torch.zeros_like(mask, dtype=torch.bool)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                near |= torch.roll(mask, (dz, dy, dx), (0, 1, 2)) != 0
    return torch.nonzero(((mask == 0) & near).reshape(-1)).reshape(-1)


class _Exact:
    """The variational problem of one cell."""

    def __init__(self, mask):
        self.nz, self.ny, self.nx = mask.shape
        self.mask = mask
        self.sup = _support(mask)
        self.nb = self.sup.numel()
        self.g = _green(self.nx, self.ny, self.nz)

    def green(self, f):
        g = self.g
        F = torch.fft.rfftn(f, dim=(1, 2, 3))
        U = torch.stack([g[0] * F[0] + g[1] * F[1] + g[2] * F[2], g[1] * F[0] + g[3] * F[1] + g[4] * F[2],
                         g[2] * F[0] + g[4] * F[1] + g[5] * F[2]])
        return torch.fft.irfftn(U, s=(self.nz, self.ny, self.nx), dim=(1, 2, 3))

    def scatter(self, x):
        f = torch.zeros((3, self.mask.numel()), dtype=torch.float64, device="cuda")
        f[:, self.sup] = (x - x.mean(0)).T
        return f.reshape(3, self.nz, self.ny, self.nx)

    def gather(self, u):
        y = u.reshape(3, -1)[:, self.sup].T
        return y - y.mean(0)

    def apply(self, x):
        return self.gather(self.green(self.scatter(x)))

    def f0(self, grad):
        f = torch.zeros((3, self.mask.numel()), dtype=torch.float64, device="cuda")
        fluid = (self.mask != 0).reshape(-1)
        nf = int(fluid.sum())
        for c in range(3):
            f[c, fluid] = -grad[c]
            f[c, self.sup] = -grad[c] * nf / self.nb
        return f.reshape(3, self.nz, self.ny, self.nx)

    def rhs(self, grad):
        return -self.gather(self.green(self.f0(grad)))

    def recover(self, grad, x):
        u = self.green(self.f0(grad) + self.scatter(x))
        v = u - u.reshape(3, -1)[:, self.sup].mean(1)[:, None, None, None]
        return v.reshape(3, -1).mean(1), v

    def tensor(self, tol=1e-12):
        """K by conjugate gradients on the mean-free forces."""
        K = torch.zeros((3, 3), dtype=torch.float64, device="cuda")
        for col in range(3):
            grad = [1.0 if c == col else 0.0 for c in range(3)]
            b = self.rhs(grad)
            x, r = torch.zeros_like(b), b.clone()
            p, rr = r.clone(), float((r * r).sum())
            stop = tol * tol * rr
            for _ in range(8000):
                if rr <= stop:
                    break
                Ap = self.apply(p)
                a = rr / float((p * Ap).sum())
                x += a * p
                r -= a * Ap
                new = float((r * r).sum())
                p = r + (new / rr) * p
                rr = new
            K[:, col] = self.recover(grad, x)[0]
        return K


def _exact_brinkman(mask, iterations):
    """The relaxed-Jacobi momentum step and 35-sweep projection of the reference."""
    fluid = mask != 0

    def sh(a, d, s):
        return torch.roll(a, s, 2 - d)

    def nbr(a):
        return sh(a, 0, 1) + sh(a, 0, -1) + sh(a, 1, 1) + sh(a, 1, -1) + sh(a, 2, 1) + sh(a, 2, -1)

    def grad(a, d):
        return 0.5 * (sh(a, d, -1) - sh(a, d, 1))

    den = torch.where(fluid, 6.0, 1.0e8 + 6.0).double()
    u = [torch.zeros(mask.shape, dtype=torch.float64, device="cuda") for _ in range(3)]
    p = torch.zeros_like(u[0])
    for _ in range(iterations):
        s = [0.9 * (((1.0 if d == 0 else 0.0) - grad(p, d) + nbr(u[d])) / den) + (1.0 - 0.9) * u[d] for d in range(3)]
        div = grad(s[0], 0) + grad(s[1], 1) + grad(s[2], 2)
        phi = torch.zeros_like(p)
        for _ in range(35):
            phi = (nbr(phi) - div) / 6.0
        u = [s[d] - grad(phi, d) for d in range(3)]
        p = p + phi
    U = torch.stack([x.mean() for x in u])
    return [U, u[0], u[1], u[2], p, None]


def _exact_conv(case, seed):
    x, dy, w, b = _conv_inputs(case, seed)
    e, s, cin, cout = case["edge"], case["samples"], case["cin"], case["cout"]
    x = x.double().reshape(s, e, e, e, cin)
    dy64 = dy.double().reshape(s, e, e, e, cout)
    w = w.double()
    y = torch.zeros_like(dy64) + b.double()
    dx = torch.zeros_like(x)
    dw = torch.zeros((27, cout, cin), dtype=torch.float64, device="cuda")
    for tap in range(27):
        off = tap // 9 - 1, tap // 3 % 3 - 1, tap % 3 - 1
        xs = torch.roll(x, tuple(-o for o in off), (1, 2, 3))
        y += xs @ w[tap].T
        dw[tap] = dy64.reshape(-1, cout).T @ xs.reshape(-1, cin)
        dx += torch.roll(dy64, off, (1, 2, 3)) @ w[tap]
    return [y.relu().reshape(-1, cout), dx.reshape(-1, cin), dw, dy64.reshape(-1, cout).sum(0)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "conv":
        return _exact_conv(case, seed)
    if kind in ("batch", "fixed"):
        return None
    mask = _mask(case, seed)
    if kind == "brinkman":
        return _exact_brinkman(mask, case["iterations"])
    if kind == "solve" and mask.numel() > 64 ** 3:
        return None  # the FP64 solve of a large cell takes too long
    ex = _Exact(mask)
    if kind == "solve":
        return ex.tensor()
    x = _vector(3 * ex.nb, seed).reshape(-1, 3)
    if kind == "apply":
        return ex.apply(x).reshape(-1)
    avg, v = ex.recover(GRAD, x)
    return [ex.rhs(GRAD).reshape(-1), avg, v]
