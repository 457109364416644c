"""The 64-byte nodes that large trees are walked through (csrc/walk_nodes.h),
checked on the host by small C++ programs compiled against the headers the
kernels use."""
from __future__ import annotations

import os
import shutil
import subprocess
from fractions import Fraction

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

PLANES = COMMON + r"""
static uint32_t state = 7;
static uint32_t bits() { return (state = state * 1664525u + 1013904223u) >> 8; }
// A float of any sign and of a magnitude between 2^-140 and 2^49.
static float any_float(int span) {
    const float m = 1.0f + (float)bits() / 16777216.0f;
    const int e = (int)(bits() % 190u) * span / 100 - 140 * span / 100;
    return ldexpf((bits() & 1u) ? m : -m, e);
}

int main() {
    for (int k = 0; k < 4000; ++k) {
        float lo[4], hi[4];
        int32_t link[4];
        const int span = 1 + (int)(bits() % 100u);  // how many magnitudes the node mixes
        for (int c = 0; c < 4; ++c) {
            link[c] = c < 2 || (bits() & 1u) ? ~c - 8 : ~0;
            lo[c] = any_float(span);
            hi[c] = any_float(span);
            if (k % 3 == 0) hi[c] = 1.0f;
            if (k % 5 == 0) lo[c] = 0.0f;
            if (lo[c] > hi[c]) std::swap(lo[c], hi[c]);
        }
        if (k == 0) lo[0] = -1e-20f, hi[0] = 1.0f, lo[1] = hi[1] = 1.0f, link[2] = link[3] = ~0;
        float origin, step;
        uint32_t ql, qh;
        walk_axis(lo, hi, link, origin, step, ql, qh);
        for (int c = 0; c < 4; ++c)
            if (link[c] != ~0)
                printf("%a %a %a %a %u %u\n", lo[c], hi[c], origin, step, (ql >> (8 * c)) & 255u, (qh >> (8 * c)) & 255u);
    }
    printf("OK\n");
    return 0;
}
"""

ENTRIES = COMMON + r"""
static uint32_t state = 11;
static float u01() { return (float)((state = state * 1664525u + 1013904223u) >> 8) / 16777216.0f; }
static float sym() { return 2.0f * u01() - 1.0f; }
static float size(float lo, float hi) { return exp2f(lo + (hi - lo) * u01()); }

int main() {
    int errors = 0, hits = 0;
    for (int k = 0; k < 200000; ++k) {
        // a node of 2^-16 to 2^8 around a point up to 2^8 away, flat on an axis now and then
        float w[32];
        int32_t link[4];
        const float extent = size(-16.0f, 8.0f), away = size(-8.0f, 8.0f);
        float mid[3];
        for (int a = 0; a < 3; ++a) {
            mid[a] = sym() * away;
            const bool flat = u01() < 0.1f;
            for (int c = 0; c < 4; ++c) {
                const float p = mid[a] + sym() * extent, q = p + u01() * extent * size(-12.0f, 0.0f);
                w[8 * a + c] = flat ? mid[a] : p;
                w[8 * a + 4 + c] = flat ? mid[a] : q;
            }
        }
        for (int c = 0; c < 4; ++c) link[c] = ~(8 * (c + 1));
        memcpy(w + 24, link, 16);
        const WalkBoxes b = boxes_of(w);
        // rays towards points of the node's boxes, corners and faces among them, from near and far
        const int c = k & 3;
        float target[3], d[3];
        const float dist = extent * size(-4.0f, 22.0f);
        for (int a = 0; a < 3; ++a) {
            const float s = u01();
            const float lo = w[8 * a + c], hi = w[8 * a + 4 + c];
            target[a] = s < 0.3f ? lo : s < 0.6f ? hi : lo + (hi - lo) * u01();
            d[a] = sym() * (u01() < 0.2f ? 1e-9f : 1.0f) * (u01() < 0.1f ? 0.0f : 1.0f);
        }
        const float scale = size(-20.0f, 20.0f);
        const RayPre ray = make_ray(mk(target[0] - d[0] * dist, target[1] - d[1] * dist, target[2] - d[2] * dist),
                                    mk(d[0] * scale, d[1] * scale, d[2] * scale));
        const float tfar = u01() < 0.5f ? INFINITY : dist / scale * (0.99f + 0.02f * u01());
        float t[4];
        walk_entries(b, ray, tfar, t);
        for (int j = 0; j < 4; ++j) {
            const float e = slab_entry(w[j], w[4 + j], w[8 + j], w[12 + j], w[16 + j], w[20 + j], ray, tfar);
            hits += e != INFINITY;
            if (e != INFINITY && !(t[j] <= e)) ++errors;  // accepted, and entered no later
        }
    }
    printf("%d boxes entered\n", hits);
    if (hits < 100000) ++errors;
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
    return out.stdout


def test_trees_whose_walk_could_overflow_the_stack_get_no_walk_nodes(tmp_path):
    """A ray from far away enters the empty slots too: three entries a node."""
    run(tmp_path, STACK)


def test_walk_boxes_contain_the_boxes(tmp_path):
    """Exactly, also where planes of very different magnitudes share a node."""
    lines = run(tmp_path, PLANES).split("\n")
    checked = 0
    for line in lines:
        f = line.split()
        if len(f) != 6:
            continue
        lo, hi, origin, step = (Fraction(float.fromhex(x)) for x in f[:4])
        ql, qh = int(f[4]), int(f[5])
        assert origin + ql * step / 2**15 <= lo <= hi <= origin + qh * step / 2**15, line
        checked += 1
    assert checked > 8000


def test_walk_boxes_are_entered_wherever_the_boxes_are(tmp_path):
    """A ray that the exact box test accepts is accepted, at no later distance."""
    run(tmp_path, ENTRIES)
