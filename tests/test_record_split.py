"""The brute-force hitters' split of their records into ranges
(split_records, csrc/kernels.h): whole tiles that cover every record once,
within the grid's limit, also for no records at all (a scene of the sentinel
alone).  The header's host form is compiled here and checked on the CPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r'''
#include <cstdio>
#include "kernels.h"
using namespace splat;
int main() {
    const long long sizes[] = {0, 1, 31, 32, 33, 64, 255, 256, 257, 1000, 20482, 96012, 1 << 24, 1 << 27};
    const long long wants[] = {1, 2, 7, 152, 4864, 70000, 1000000};
    const long long tiles[][2] = {{32, 32}, {64, 64}, {256, 64}, {128, 128}, {256, 256}};  // least, tile
    for (long long n : sizes)
        for (long long want : wants)
            for (auto& t : tiles) {
                const RecordSplit r = split_records(n, want, t[0], t[1]);
                const bool ok = r.splits >= 1 && r.splits <= 65535 && r.splits <= want && r.per_split >= t[1] &&
                                r.per_split % t[1] == 0 && r.splits * r.per_split >= n &&
                                (r.splits == 1 || (r.splits - 1) * r.per_split < n);
                if (!ok) {
                    std::printf("n %lld want %lld tile %lld: %lld x %lld\n", n, want, t[1], (long long)r.splits,
                                (long long)r.per_split);
                    return 1;
                }
            }
    std::printf("ok\n");
    return 0;
}
'''


def test_records_are_split_into_whole_tiles(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    src = tmp_path / "record_split_check.cu"
    src.write_text(SOURCE)
    exe = tmp_path / "record_split_check"
    inc = os.path.join(ROOT, "splat_gb300", "csrc")
    r = subprocess.run([nvcc, "-O2", "-std=c++17", "-I", inc, "-I", os.path.join(ROOT, "include"), str(src), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", (out.returncode, out.stdout + out.stderr)
