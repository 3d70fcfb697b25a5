"""The group traversal's shared-memory stack (group_take, group_fits in
csrc/hitcore.cuh) stays within its entries whatever the tree: a step takes
off what leaves room for its children, and where a tree is deeper than the
host builder makes one (a rebuilt one may be) the step that would run past
the end is told so.  The header's host forms are compiled here and run over
trees whose every box is entered, on the CPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r'''
#include <cstdio>
#include <random>
#include <vector>
#include "hitcore.cuh"
using namespace splat;

// Walks a tree of `depth` levels of inner nodes; an inner node has 4 children
// (full) or 0 to 4 at random, a leaf none.  Returns the most entries held, -1
// when a push would have run past the stack; told: a step was refused.
template <int G>
int walk(int depth, bool full, unsigned seed, long steps, bool& told) {
    std::mt19937 rng(seed);
    std::vector<int> stack(kGroupStack<G>, 0);
    int sp = 1, most = 1;
    stack[0] = depth;
    told = false;
    for (long i = 0; i < steps && sp > 0; ++i) {
        const int take = group_take<G>(sp);
        if (take < 1 || take > G || take > sp) return -2;
        std::vector<int> mine(stack.begin() + (sp - take), stack.begin() + sp);
        sp -= take;
        const bool fits = group_fits<G>(sp, take);
        if (!fits) told = true;
        for (int d : mine) {
            if (d == 0 || !fits) continue;
            const int children = full ? 4 : (int)(rng() % 5u);
            for (int c = 0; c < children; ++c) {
                if (sp >= kGroupStack<G>) return -1;
                stack[sp++] = full || rng() % 3u ? d - 1 : 0;
            }
        }
        if (sp > most) most = sp;
    }
    return most;
}

template <int G>
bool check() {
    const int bound = (kBvhStack - 2) / 3;  // the host builder's: 3 levels + 1 < kBvhStack
    for (int depth = 1; depth <= 61; ++depth)
        for (unsigned seed = 0; seed < 12; ++seed) {
            bool told;
            const int most = walk<G>(depth, seed == 0, seed, 200000, told);
            if (most < 0 || most > kGroupStack<G> || (told && depth <= bound)) {
                std::printf("G %d depth %d seed %u: %d told %d\n", G, depth, seed, most, (int)told);
                return false;
            }
            if (seed == 0 && depth == 61 && !told) {
                std::printf("G %d: a full tree of 61 levels was not refused\n", G);
                return false;
            }
        }
    return true;
}

int main() {
    if (!check<8>() || !check<32>()) return 1;
    std::printf("ok\n");
    return 0;
}
'''


def test_group_stack_stays_in_bounds(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    src = tmp_path / "group_stack_check.cu"
    src.write_text(SOURCE)
    exe = tmp_path / "group_stack_check"
    inc = os.path.join(ROOT, "splat_gb300", "csrc")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "-I", inc, "-I",
                        os.path.join(ROOT, "include"), str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
