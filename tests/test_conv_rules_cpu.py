"""The rule that chooses the convolution's form (csrc/conv_rules.h) in a host
program: every choice is one the kernels take, the choices at measured calls are
the measured better side, and the sizes of the GPU test reach every form."""
import ctypes as C
import os
import random
import shutil
import subprocess

import pytest

from conftest import ROOT

SOURCE = r"""
#include "conv_rules.h"
extern "C" void plan(const long long* size, const int* c, long long* out) {
    const fp::ConvCall call{size[0], size[1], size[2], size[3], c[0], c[1], c[2], c[3]};
    const fp::ConvPlan p = fp::conv_plan(call);
    const std::size_t smem = p.halo ? fp::conv_halo_smem(call.nx, call.cin, p.tile)
                                    : fp::conv_tap_smem(call.cin, p.tile, p.stages);
    out[0] = p.halo;
    out[1] = p.tile;
    out[2] = p.stages;
    out[3] = (long long)smem;
    out[4] = fp::conv_residents(smem);
    out[5] = p.halo ? fp::conv_halo_grid(call, p.tile) : 0;
    out[6] = p.halo && !fp::conv_halo_ok(call, p.tile);
    out[7] = fp::conv_halo_tiles(call);
}
"""

# (tile form, output channels per CTA, buffers): (nx, ny, nz, samples, cin, cout, dilation)
FORMS = {
    (1, 16, 0): (1, 1, 1, 1, 16, 16, 1),
    (1, 32, 0): (1, 1, 1, 22, 64, 128, 1),
    (1, 64, 0): (1, 1, 1, 47, 16, 128, 1),
    (1, 128, 0): (3, 3, 1, 116, 16, 128, 1),
    (0, 16, 2): (2, 85, 46, 5, 112, 16, 1),
    (0, 16, 3): (1, 6, 10, 325, 112, 16, 2),
    (0, 16, 4): (1, 1, 1, 1, 16, 32, 2),
    (0, 32, 2): (1, 19, 38, 27, 128, 32, 2),
    (0, 32, 3): (3, 12, 2, 271, 112, 32, 1),
    (0, 32, 4): (14, 3, 29, 2, 112, 128, 2),
    (0, 64, 2): (3, 7, 103, 9, 112, 64, 1),
    (0, 64, 3): (2, 16, 4, 153, 96, 64, 2),
    (0, 64, 4): (3, 1, 2, 811, 16, 128, 2),
    (0, 128, 2): (16, 4, 5, 61, 80, 128, 1),
    (0, 128, 3): (14, 29, 8, 3, 128, 128, 1),
    (0, 128, 4): (1, 29, 24, 14, 48, 128, 2),
}


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("conv")
    (d / "rules.cpp").write_text(SOURCE)
    so = str(d / "rules.so")
    subprocess.run([gxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "fft_method_test_gb300", "csrc"), "-o", so, str(d / "rules.cpp")], check=True)
    lib = C.CDLL(so)

    def call(nx, ny, nz, samples, cin, cout, dil=1, sms=152):
        out = (C.c_longlong * 8)()
        lib.plan((C.c_longlong * 4)(nx, ny, nz, samples), (C.c_int * 4)(dil, cin, cout, sms), out)
        return list(out)

    return call


def test_every_choice_is_a_form_the_kernels_have(plan):
    rng = random.Random(3)
    for _ in range(20000):
        n = [int(2 ** rng.uniform(0, rng.choice((3, 8, 13)))) for _ in range(3)]
        samples = int(2 ** rng.uniform(0, 14))
        if n[0] * n[1] * n[2] * samples > 2 ** 37:
            continue
        cin, cout = 16 * rng.randint(1, 8), rng.choice((16, 32, 64, 128))
        dil, sms = rng.choice((1, 1, 2, 5)), rng.choice((152, 152, 20, 1))
        halo, tile, stages, smem, residents, grid, bad, tiles = plan(*n, samples, cin, cout, dil, sms)
        assert tile in (16, 32, 64, 128) and cout % tile == 0 and tile <= cout
        assert smem <= 232448
        assert residents * max(32, tile) <= 512  # tensor-memory columns of an SM
        if halo:
            assert not bad and dil == 1 and cin <= 64 and 1 <= grid <= tiles
            assert 3 * (128 + 2 * (n[0] + 3)) <= 0x3FFF
        else:
            assert stages in (2, 3, 4)


@pytest.mark.parametrize("size,halo,tile", [
    # the tile form where its rows are fewer
    ((32, 32, 32, 4, 16, 32), 1, 32), ((4, 4, 4, 4, 64, 128), 1, None), ((64, 64, 64, 2, 16, 16), 1, 16),
    # not on samples smaller than a tile, thin cells, long rows, many splits
    ((1, 1, 1, 4096, 64, 64), 0, None), ((2, 2, 2, 1024, 64, 128), 0, None), ((4, 4, 4, 512, 64, 128), 0, None),
    ((1000, 16, 16, 1, 16, 32), 0, 32), ((64, 1, 64, 16, 64, 128), 0, 128), ((64, 64, 64, 2, 64, 128), 0, 128),
    # all output channels in a CTA once the voxels alone fill the SMs, fewer before
    ((16, 16, 16, 4, 128, 128), 0, 128), ((8, 8, 8, 4, 128, 128), 0, 16)])
def test_measured_calls_take_their_better_side(plan, size, halo, tile):
    out = plan(*size)
    assert out[0] == halo and (tile is None or out[1] == tile), out


def test_sizes_of_the_gpu_test_reach_every_form(plan):
    for form, size in FORMS.items():
        assert tuple(plan(*size)[:3]) == (form if form[0] else (0, form[1], form[2])), (form, size)
