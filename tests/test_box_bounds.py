"""The box around eight blocks of the finder (csrc/boxes.h, as k_prepare combines it over a
shuffle tree): it holds every block, and a block whose box is no number, because its first
atom's position is none, takes no other block out of the lists."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openmm-atmmetaforce-plugin_gb300",
                    "csrc")

PROGRAM = r"""
#include <cstdio>
#include <limits>
#include "boxes.h"
using namespace atm;

// one axis: the octet's centre and half extent from eight blocks' (offset, half extent)
static void octet(const float* d, const float* h, float& c, float& e) {
    float lo[8], hi[8];
    for (int k = 0; k < 8; k++) {
        lo[k] = d[k] - h[k];
        hi[k] = d[k] + h[k];
    }
    for (int o = 1; o <= 4; o <<= 1) {
        float l2[8], h2[8];
        for (int k = 0; k < 8; k++) {
            l2[k] = bound_min(lo[k], lo[k ^ o]);
            h2[k] = bound_max(hi[k], hi[k ^ o]);
        }
        for (int k = 0; k < 8; k++) {
            lo[k] = l2[k];
            hi[k] = h2[k];
        }
    }
    c = 0.5f * (lo[0] + hi[0]);
    e = 0.5f * (hi[0] - lo[0]);
}

int main() {
    const float nan = std::numeric_limits<float>::quiet_NaN(), inf = std::numeric_limits<float>::infinity();
    const float cut2 = 0.81f;
    const float d0[8] = {0.f, 0.2f, -0.3f, 0.5f, 0.1f, -0.1f, 0.4f, 0.3f}, h0[8] = {.2f, .1f, .3f, .2f, .25f, .2f, .1f, .3f};
    float c, e;
    octet(d0, h0, c, e);
    for (int k = 0; k < 8; k++)
        if (d0[k] - h0[k] < c - e - 1e-6f || d0[k] + h0[k] > c + e + 1e-6f) return printf("a block outside\n"), 1;
    // a row far away on this axis: out of reach of the numbers, within reach of none
    const float row = 5.0f, rh = 0.3f;
    if (box_gap2(c - row, 0.f, 0.f, rh + e, rh, rh) < cut2) return printf("far octet kept\n"), 1;
    const float none[3] = {nan, inf, -inf};
    for (float bad : none)
        for (int k = 0; k < 8; k++) {
            float d[8], h[8];
            for (int q = 0; q < 8; q++) {
                d[q] = d0[q];
                h[q] = h0[q];
            }
            d[k] = bad;
            if (bad != bad) h[k] = bad;
            octet(d, h, c, e);
            if (box_gap2(c - row, 0.f, 0.f, rh + e, rh, rh) >= cut2) return printf("block %d dropped its octet\n", k), 1;
        }
    return 0;
}
"""


def test_octets_of_blocks_hold_what_is_no_number(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "octets.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "octets"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
