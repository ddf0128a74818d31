"""How many sectors a launch of the split sweep takes, on the CPU: the rule of the library
and of its header."""

import shutil
import subprocess
from pathlib import Path

from conftest import PKG_DIR


def test_a_shorter_run_keeps_the_planes_of_the_whole_one(tmp_path):
    """Planes are sized for 180 sectors in launches of even size.  A run of fewer sectors,
    as the autotuner's, may want more of them in a launch: it takes what there is, in
    launches of even size, and adds surfaces in turn only where not one sector's fit."""
    main, exe = tmp_path / "main.cpp", tmp_path / "main"
    main.write_text(r"""
#include <cstdio>
#include <cuda_runtime.h>
#include "tvs_internal.cuh"
int main() {
    const int mixed64 = 1;
    const tvs::QueueConfig quad{4, 1, 0, 0, 9};
    int shorter = 0;
    for (uint32_t tiles = 1; tiles < 40000; tiles += 1 + tiles / 50) {
        uint32_t whole = 0;
        const size_t held = tvs::split_plane_bytes(mixed64, quad, tiles, 180, &whole);
        if (tvs::plane_sectors(held, held, whole, 180) != whole) return 1;
        for (uint32_t n = 1; n <= 180; n++) {
            uint32_t want = 0;
            const size_t bytes = tvs::split_plane_bytes(mixed64, quad, tiles, n, &want);
            const uint32_t per = tvs::plane_sectors(held, bytes, want, n);
            shorter += bytes > held;
            if (per == 0 || per > n || (size_t)per * (bytes / want) > held) return 2;
            if (bytes <= held && per != want) return 3;
        }
    }
    if (shorter == 0) return 4;  // the case is there: 32 sectors fit, 180 take 30 a launch
    if (tvs::plane_sectors(0, 4096, 4, 4) != 0 || tvs::plane_sectors(1023, 4096, 4, 4) != 0) return 5;
    if (tvs::plane_sectors(1024, 4096, 4, 4) != 1 || tvs::plane_sectors(1 << 20, 0, 0, 4) != 0) return 6;
    return 0;
}
""")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([shutil.which("g++"), "-std=c++17", "-O1", "-w", "-I", str(PKG_DIR / "csrc"), "-I",
                    str(PKG_DIR.parent / "include"), "-I",
                    str(Path(nvcc).resolve().parent.parent / "include"), str(main), "-L", str(PKG_DIR),
                    "-ltvs_cuda", f"-Wl,-rpath,{PKG_DIR}", "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
