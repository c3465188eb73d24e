"""The launch rules of csrc/launch_rules.h in a host program, with stand-ins for
the CUDA calls: what a process with a second device, or a device that cannot
place a large cluster, gets, and which failures of a lockstep solve are tried again
one case at a time."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

MAIN = r"""
#include <cstdio>
#include "launch_rules.h"

// device d allows 16-block clusters when bit 0 of caps[d] is set and can place
// clusters of up to caps[d] / 2 blocks
static int caps[4] = {33, 33, 32, 9};
static bool allowed[4];
static int asked;

static int blocks(std::atomic<int> (&known)[fp::kClusterDevices], int dev) {
    return fp::cluster_blocks(
        known, dev,
        [&] { return ++asked, allowed[dev] = caps[dev] & 1; },
        [&](int n) { return n <= caps[dev] / 2 && (n <= 8 || allowed[dev]); });
}

int main() {
    static std::atomic<int> known[fp::kClusterDevices];
    for (int turn = 0; turn < 2; ++turn)
        for (int dev = 0; dev < 4; ++dev) std::printf("%d ", blocks(known, dev));
    std::printf("%d", asked);
    static std::atomic<int> none[fp::kClusterDevices];
    std::printf(" %d", fp::cluster_blocks(none, 200, [] { return true; }, [](int) { return false; }));
    // {code, an allocation failed}: done, a device error, no memory (two codes), not converged
    const int codes[][2] = {{0, 0}, {3, 0}, {3, 1}, {5, 1}, {2, 0}};
    for (auto& c : codes) {
        int again = 0;
        const int rc = fp::lockstep_or_one_by_one(
            [&](bool* no_memory) { return *no_memory = c[1], c[0]; }, [&] { return ++again, 0; });
        std::printf(" %d%d", rc, again);
    }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("rules")
    (d / "main.cpp").write_text(MAIN)
    exe = str(d / "rules")
    subprocess.run([gxx, "-std=c++17", "-I", os.path.join(ROOT, "fft_method_test_gb300", "csrc"), "-o", exe,
                    str(d / "main.cpp")], check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout


def test_cluster_blocks_belong_to_their_device(program):
    out = [int(v) for v in program.split()]
    assert out[:4] == [16, 16, 8, 4]  # each device's own attribute and room
    assert out[4:8] == out[:4]
    assert out[8] == 4  # the attribute is set once on each device
    assert out[9] == 1  # beyond the table, and no cluster fits


def test_bias_gradient_keeps_no_process_wide_attribute():
    src = open(os.path.join(ROOT, "fft_method_test_gb300", "csrc", "learned.cu")).read()
    body = src[src.index("fp_nn_bias_grad("):]
    body = body[:body.index("\n}")]
    assert "cluster_blocks(" in body and "static const bool" not in body


def test_only_a_lack_of_memory_is_tried_again(program):
    assert program.split()[10:] == ["00", "30", "01", "01", "20"]
