"""Which device arrays share a copy to the host (csrc/gsofa_fetch.h), on the
CPU: arrays of one allocation may, arrays of different allocations may not,
whatever lies between them; and the staged arrays hold what the device arrays
hold."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "gsofa_fetch.h"
using namespace gsofa::host;

static char device[1 << 16];
static int checks = 0;

static void check(bool ok, const char* what, int i) {
    checks++;
    if (ok) return;
    std::printf("%s (%d)\n", what, i);
    std::exit(1);
}

int main() {
    for (size_t i = 0; i < sizeof device; i++) device[i] = (char)(i * 131 >> 3);
    std::srand(7);
    for (int round = 0; round < 20000; round++) {
        // allocations of 256-byte steps side by side, some of them of two or three arrays
        Fetch f[kMaxFetch];
        int owner[kMaxFetch], count = 0, id = 0;
        size_t at = 0, begin[kMaxFetch], end[kMaxFetch];
        char out[kMaxFetch][1024];
        while (count < 6) {
            const int arrays = 1 + std::rand() % 3;
            const size_t first = at;
            const int k0 = count;
            for (int a = 0; a < arrays && count < kMaxFetch; a++, count++) {
                const size_t bytes = std::rand() % 5 ? 1 + std::rand() % 900 : 0;
                f[count] = {std::rand() % 6 ? out[count] : nullptr, device + at, bytes, device + first};
                owner[count] = id;
                at += (bytes + kFetchStep - 1) / kFetchStep * kFetchStep;
                if (std::rand() % 4 == 0) at += 512;  // an array that was not asked for
            }
            for (int k = k0; k < count; k++) begin[k] = first, end[k] = at;
            if (arrays == 1 && std::rand() % 2) f[k0].block = nullptr;
            id++;
        }
        const FetchPlan p = plan_fetch(f, count);
        char stage[1 << 16];
        size_t used = 0;
        for (int c = 0; c < p.copies; c++) {
            const size_t a = p.copy[c].src - device, b = a + p.copy[c].bytes;
            int touched = -1;
            for (int k = 0; k < count; k++) {
                if (b <= begin[k] || a >= end[k]) continue;
                check(touched < 0 || touched == owner[k], "a copy spans two allocations", round);
                touched = owner[k];
                check(a >= begin[k] && b <= end[k], "a copy leaves its allocation", round);
            }
            check(p.copy[c].at >= used, "staged copies overlap", round);
            used = p.copy[c].at + p.copy[c].bytes;
            std::memcpy(stage + p.copy[c].at, p.copy[c].src, p.copy[c].bytes);
        }
        check(used <= p.bytes, "the staging buffer is larger than said", round);
        size_t total = 0;
        for (int k = 0; k < count; k++) {
            if (!f[k].dst || !f[k].bytes) continue;
            total += f[k].bytes;
            check(!std::memcmp(stage + p.at[k], f[k].src, f[k].bytes), "an array differs", round);
        }
        check(p.bytes <= total + kFetchStep * (size_t)count, "more staging than the bound", round);
    }
    // three arrays of one allocation are one copy, of three allocations three
    Fetch g[3] = {{device, device, 200, device}, {device, device + 256, 200, device}, {device, device + 512, 9, device}};
    check(plan_fetch(g, 3).copies == 1, "one allocation", 0);
    for (Fetch& x : g) x.block = x.src;
    check(plan_fetch(g, 3).copies == 3, "three allocations", 0);
    for (Fetch& x : g) x.block = nullptr;
    check(plan_fetch(g, 3).copies == 3, "allocations of their own", 0);
    std::printf("%d\n", checks);
    return 0;
}
"""


def test_copies_stay_inside_one_allocation(tmp_path):
    src, exe = tmp_path / "fetch.cpp", tmp_path / "fetch"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "gsofatpds_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert int(out.stdout) > 100000
