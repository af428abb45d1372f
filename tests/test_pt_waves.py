"""How a render's samples and pixels fall into waves (pt_wave.h): host code, compiled
here on its own and run with the figures that the path tracer passes."""
import os
import subprocess

import pytest

from conftest import ROOT

CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
pytestmark = pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")), reason="no CUDA headers")


def run(tmp_path, body):
    src, exe = tmp_path / "waves.cpp", tmp_path / "waves"
    src.write_text('#include <climits>\n#include <cstdio>\n#include <cstdlib>\n#include <vector>\n#include "pt_wave.h"\n'
                   "#define CHECK(x) do { if (!(x)) { std::printf(\"%d: %s\\n\", __LINE__, #x); return 1; } } while (0)\n"
                   "using namespace sg;\n" + body)
    csrc = os.path.join(ROOT, "sort_b200", "csrc")
    r = subprocess.run(["g++", "-std=c++17", "-ftrapv", "-Wall", "-I" + csrc, "-I" + os.path.join(ROOT, "include"),
                        "-I" + CUDA, str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_waves_hold_every_sample_once(tmp_path):
    """Also for sample counts next to the largest int."""
    run(tmp_path, """
int main() {
    for (int spp : {1, 2, 5, 63, 65535, (1 << 20) - 1, 1 << 20, (1 << 20) + 1, INT_MAX - 1, INT_MAX})
        for (long pixels : {1l, 3l, 14651l, (1l << 20) - 1, 1l << 20, 1l << 27}) {
            const int per = wave_samples(pixels, kWavePaths, spp), waves = wave_count(spp, per);
            CHECK(per >= 1 && per <= spp && waves >= 1);
            CHECK(long(waves) * per >= spp && long(waves - 1) * per < spp);
            CHECK(per == 1 || pixels * per <= kWavePaths);
        }
    CHECK(wave_count(INT_MAX, 1 << 20) == 2048);
}
""")
