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


def test_memory_of_waves(tmp_path):
    """Samples that share waves take no more than 64 MB or a sixteenth of the free memory
    (asked for above 64 MB only), a size that could not be had is not asked for again by the next render, and what a
    scene holds is released only for something larger, or to make room for a sample
    per wave."""
    run(tmp_path, """
struct Fake {
    size_t free = 0, held = 0;
    size_t limit = SIZE_MAX;  // the largest single allocation
    cudaError_t error = cudaErrorMemoryAllocation;
    std::vector<size_t> asked, live;
    int released = 0;
    int asked_free = 0;
    size_t free_bytes() { ++asked_free; return free; }
    cudaError_t alloc(size_t bytes, char** mem) {
        asked.push_back(bytes);
        if (bytes > free || bytes > limit) return error;
        *mem = static_cast<char*>(std::malloc(sizeof(size_t)));
        *reinterpret_cast<size_t*>(*mem) = bytes;
        free -= bytes;
        held += bytes;
        return cudaSuccess;
    }
    void release(char* mem) {
        const size_t bytes = *reinterpret_cast<size_t*>(mem);
        std::free(mem);
        free += bytes;
        held -= bytes;
        ++released;
    }
};
const size_t GiB = size_t(1) << 30, MiB = size_t(1) << 20;

int main() {
    WavePlan p;
    {  // room: as many samples as a wave takes; the next render allocates nothing
        Fake g;
        g.free = 170 * GiB;
        WaveBuffers b;
        CHECK(fit_wave_buffers(g, b, 64 * 64, 4096, p) == cudaSuccess);
        CHECK(p.per_wave == 256 && p.waves == 16 && p.in_flight == 2 && p.bytes <= 425 * size_t(1000000));
        CHECK(b.bytes == p.bytes && g.asked.size() == 1);
        CHECK(fit_wave_buffers(g, b, 64 * 64, 4096, p) == cudaSuccess && p.per_wave == 256);
        CHECK(fit_wave_buffers(g, b, 61, 4096, p) == cudaSuccess && g.asked.size() == 1 && g.released == 0);
        CHECK(g.asked_free == 1);
        WaveBuffers c;  // a small one is not worth asking
        g.free = 100 * MiB;
        CHECK(fit_wave_buffers(g, c, 161 * 91, 4, p) == cudaSuccess && p.per_wave == 4 && g.asked_free == 1);
        CHECK(fit_wave_buffers(g, c, 64 * 64, 4096, p) == cudaSuccess && c.bytes <= 64 * MiB && c.bytes > 32 * MiB);
    }
    {  // little room: at most a sixteenth of it, and no attempt at more
        Fake g;
        g.free = 2 * GiB;
        WaveBuffers b;
        CHECK(fit_wave_buffers(g, b, 64 * 64, 4096, p) == cudaSuccess);
        CHECK(p.per_wave > 1 && b.bytes <= 128 * MiB && g.asked.size() == 1);
        const size_t held = b.bytes;
        g.free = 170 * GiB;
        CHECK(fit_wave_buffers(g, b, 64 * 64, 4096, p) == cudaSuccess);
        CHECK(b.bytes == held && g.asked.size() == 1 && g.released == 0);
    }
    {  // allocations fail above 100 MiB: fewer samples share a wave, remembered by the next renders
        Fake g;
        g.free = 170 * GiB;
        g.limit = 100 * MiB;
        WaveBuffers b;
        CHECK(fit_wave_buffers(g, b, 64 * 64, 4096, p) == cudaSuccess);
        CHECK(p.per_wave > 1 && p.bytes <= 100 * MiB && p.bytes == b.bytes);
        const size_t asked = g.asked.size();
        const char* mem = b.mem;
        for (int k = 0; k < 3; ++k) {
            CHECK(fit_wave_buffers(g, b, 64 * 64, 4096, p) == cudaSuccess);
            CHECK(g.asked.size() == asked && g.released == 0 && b.mem == mem);
        }
    }
    {  // a larger frame: the old memory goes once the new one is there
        Fake g;
        g.free = 170 * GiB;
        WaveBuffers b;
        CHECK(fit_wave_buffers(g, b, 64, 2, p) == cudaSuccess && p.waves == 1);
        CHECK(fit_wave_buffers(g, b, 500000, 4, p) == cudaSuccess && p.per_wave == 2);
        CHECK(g.released == 1 && g.held == b.bytes);
        // a sample per wave may need the old memory's room
        g.free = wave_plan(1 << 27, 8, 1).bytes - b.bytes;
        CHECK(fit_wave_buffers(g, b, 1 << 27, 8, p) == cudaSuccess && p.per_wave == 1 && g.released == 2 && g.free == 0);
    }
    {  // not even that: the error, and nothing held
        Fake g;
        g.free = MiB;
        WaveBuffers b;
        CHECK(fit_wave_buffers(g, b, 1 << 20, 8, p) == cudaErrorMemoryAllocation && !b.mem && b.bytes == 0 && g.held == 0);
        g.error = cudaErrorLaunchFailure;  // another error stays itself
        CHECK(fit_wave_buffers(g, b, 1 << 16, 64, p) == cudaErrorLaunchFailure && !b.mem);
    }
    {  // frames above one wave go in parts that cover them
        const WavePlan w = wave_plan(int64_t(1) << 28, 3, 1);
        CHECK(w.parts == 2 && w.waves == 6 && w.cap == size_t(1) << 27 && int64_t(w.parts) * w.part >= int64_t(1) << 28);
    }
    return 0;
}
""")
