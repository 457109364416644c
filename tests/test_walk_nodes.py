"""The 64-byte nodes that large trees are walked through (csrc/walk_nodes.h),
checked on the host by small C++ programs compiled against the headers the
kernels use."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "aqua-engine_gb300", "csrc")

COMMON = r"""
#include "bvh.h"
#include "walk_nodes.h"
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

using namespace aq;

static RayPre make_ray(v3 o, v3 d) {
    RayPre r;
    r.o = o;
    r.invd = mk(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z));
    r.tmin = 0.0f;
    r.tmax = INFINITY;
    return r;
}

// The walk node of 32 node words: its boxes.
static WalkBoxes boxes_of(const float* w) {
    int32_t link[4];
    memcpy(link, w + 24, 16);
    WalkBoxes b;
    walk_axis(w, w + 4, link, b.ox, b.sx, b.lx, b.hx);
    walk_axis(w + 8, w + 12, link, b.oy, b.sy, b.ly, b.hy);
    walk_axis(w + 16, w + 20, link, b.oz, b.sz, b.lz, b.hz);
    return b;
}
"""

STACK = COMMON + r"""
// A chain of nodes with two children each, a leaf and the next node, in a box
// of 1e-4: max_stack as the builder counts it is one entry per node.
static FlatBvh chain(int depth) {
    FlatBvh t;
    t.depth = t.max_stack = depth;
    t.nodes.assign((size_t)kBvhNodeFloats * depth, 0.0f);
    for (int k = 0; k < depth; ++k) {
        float* w = &t.nodes[(size_t)kBvhNodeFloats * k];
        for (int a = 0; a < 3; ++a)
            for (int c = 0; c < 4; ++c) {
                w[8 * a + c] = c < 2 ? 0.0f : INFINITY;
                w[8 * a + 4 + c] = c < 2 ? 1e-4f : INFINITY;
            }
        const int32_t link[4] = {k + 1 < depth ? k + 1 : ~1, ~1, ~0, ~0};
        memcpy(w + 24, link, 16);
    }
    return t;
}

// Most stack entries of a nearest-first walk over the entry distances.
template <class Test>
static int walk(const FlatBvh& t, Test test) {
    std::vector<int32_t> stack;
    size_t most = 0;
    int32_t node = 0;
    while (true) {
        if (node >= 0) {
            const float* w = &t.nodes[(size_t)kBvhNodeFloats * node];
            int32_t link[4];
            memcpy(link, w + 24, 16);
            float e[4];
            test(w, e);
            int order[4] = {0, 1, 2, 3};
            std::stable_sort(order, order + 4, [&](int a, int b) { return e[a] < e[b]; });
            for (int k = 3; k > 0; --k)
                if (e[order[k]] != INFINITY) stack.push_back(link[order[k]]);
            most = std::max(most, stack.size());
            if (e[order[0]] != INFINITY) { node = link[order[0]]; continue; }
        }
        if (stack.empty()) return (int)most;
        node = stack.back();
        stack.pop_back();
    }
}

int main() {
    int errors = 0;
    const RayPre ray = make_ray(mk(100.0f, 100.0f, 100.0f), mk(-1.0f, -1.0f, -1.0f));
    for (int depth : {3, 31, 32, 33, 60, 95}) {
        const FlatBvh t = chain(depth);
        const int full = walk(t, [&](const float* w, float* e) {
            for (int c = 0; c < 4; ++c)
                e[c] = slab_entry(w[c], w[4 + c], w[8 + c], w[12 + c], w[16 + c], w[20 + c], ray, INFINITY);
        });
        const int wide = walk(t, [&](const float* w, float* e) { walk_entries(boxes_of(w), ray, INFINITY, e); });
        printf("depth %d: full %d, walk nodes %d, fits %d\n", depth, full, wide, (int)walk_stack_fits(t));
        if (full > t.max_stack || full >= kBvhStackSize) ++errors;     // the builder's bound holds there
        if (wide != 3 * depth) ++errors;                               // every empty slot was accepted
        if (walk_stack_fits(t) != (wide <= kBvhStackSize)) ++errors;
    }
    printf(errors ? "FAIL %d\n" : "OK\n", errors);
    return errors ? 1 : 0;
}
"""


def run(tmp_path, program):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(program)
    subprocess.run([gxx, "-std=c++17", "-O1", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip().endswith("OK"), out.stdout


def test_trees_whose_walk_could_overflow_the_stack_get_no_walk_nodes(tmp_path):
    """A ray from far away enters the empty slots too: three entries a node."""
    run(tmp_path, STACK)
