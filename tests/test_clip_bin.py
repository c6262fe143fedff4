"""clip_triangle_bin (the register form of the triangle clip for spatial bins) against the general
Sutherland-Hodgman form, on the host: wherever it takes a clip, its box has the general form's
values. Triangles and regions of every kind: vertices on planes, degenerate triangles, regions narrower
than the triangle on other axes, coordinates that are not finite."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "ray-tracer_b200", "csrc")
CUDA = "/usr/local/cuda/include"

HARNESS = r"""
#include <cmath>
#include "device_math.cuh"
#include <cstdio>
#include <random>
using namespace rtd;
int main()
{
    std::mt19937 g(1);
    auto U = [&]() { return std::uniform_real_distribution<float>(0.f, 1.f)(g); };
    long taken = 0, total = 1500000;
    for (long it = 0; it < total; it++)
    {
        const int mode = g() % 6;
        const float sc = mode == 1 ? 1e-3f : 1.f;
        f3 v[3], o = mk3(U(), U(), U());
        for (auto& p : v) { p = mk3(o.x + sc * (U() - .5f), o.y + sc * (U() - .5f), o.z + sc * (U() - .5f)); }
        if (mode == 2) { for (auto& p : v) { p = mk3(roundf(p.x * 4) / 4, roundf(p.y * 4) / 4, roundf(p.z * 4) / 4); } }
        if (mode == 3) { v[2] = v[g() % 2]; }
        box3 r = box_empty();
        for (auto& p : v) { box_pt(r, p); }
        if (mode >= 4) { for (int k = 0; k < 3; k++) { r.mn[k] -= U() * .1f; r.mx[k] += U() * .1f; } }
        if (mode == 5 && g() % 4 == 0) { r.mn[g() % 3] += .05f; }
        const float odd[4] = { NAN, INFINITY, -INFINITY, 3e38f };
        if (g() % 200 == 0) { (&v[g() % 3].x)[g() % 3] = odd[g() % 4]; }
        const int axis = g() % 3, nb = 8 + g() % 25, b = g() % nb;
        const float mn = r.mn[axis], s = nb / (r.mx[axis] - r.mn[axis]);
        r.mn[axis] = mn + (float)b / s;
        r.mx[axis] = mode == 2 && g() % 2 ? r.mn[axis] + .25f * (g() % 3) : mn + (float)(b + 1) / s;
        box3 c;
        if (!clip_triangle_bin(v[0], v[1], v[2], axis, r, c)) { continue; }
        taken++;
        const box3 e = clip_triangle_general(v[0], v[1], v[2], r);
        for (int k = 0; k < 3; k++)
        {
            if (!(c.mn[k] == e.mn[k] && c.mx[k] == e.mx[k])) { printf("mode %d axis %d: %g %g, want %g %g\n", mode, axis, c.mn[k], c.mx[k], e.mn[k], e.mx[k]); return 1; }
        }
    }
    printf("taken %ld of %ld\n", taken, total);
    return taken > total / 2 ? 0 : 2;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="needs g++ and the CUDA headers")
def test_bin_clip_equals_general_clip(tmp_path):
    src, exe = tmp_path / "clip.cpp", tmp_path / "clip"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-I", CUDA, "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
