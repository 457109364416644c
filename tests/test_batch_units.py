"""How a batch's pixels are split into work items (csrc/batch_units.h), checked
on the host: a small C++ program splits job lists, small ones and ones whose
items outgrow 32 bits, and checks that every sample of every pixel belongs to
exactly one item, and that the items' sums add up to the same bits however
the pixel was split."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "aqua-engine_gb300", "csrc")

PROGRAM = r"""
#include "batch_units.h"
#include <cmath>
#include <cstdio>

using namespace aq;

struct Job {
    int32_t spp;
    uint32_t pixels, item_begin, units, run_spp, part_begin, done_begin;
};
static Job job(uint64_t pixels, int spp) {
    Job j{};
    j.pixels = (uint32_t)pixels;
    j.spp = spp;
    j.run_spp = run_spp_of(j.pixels, (uint32_t)spp);
    return j;
}

// The pixel's value as the lanes add it up, run after run or the stored runs in order.
static float pixel_sum(const std::vector<float>& sample, const Job& j) {
    std::vector<float> part;
    float total = 0.0f;
    for (uint32_t item = 0; item < j.units; ++item) {
        const uint32_t first = item * j.run_spp;
        const uint32_t end = j.units > 1 ? std::min(first + j.run_spp, (uint32_t)j.spp) : (uint32_t)j.spp;
        for (uint32_t s = first; s < end; s += j.run_spp) {
            float sum = 0.0f;
            for (uint32_t k = s; k < std::min(s + j.run_spp, (uint32_t)j.spp); ++k) sum += sample[k];
            part.push_back(sum);
            total += sum;
        }
    }
    if (j.units == 1) return total;
    total = 0.0f;
    for (float p : part) total += p;
    return total;
}

static int check_sums() {
    int errors = 0;
    uint32_t rng = 1;
    for (int spp : {1, 2, 3, 5, 7, 8, 48, 60, 64, 255, 256, 257, 511, 1000, 4096, 5001}) {
        std::vector<float> sample((size_t)spp);
        double exact = 0.0, magnitude = 0.0;
        for (float& s : sample) {
            rng = rng * 1664525u + 1013904223u;
            s = (float)(rng >> 8) / 16777216.0f + ((rng & 63u) == 0u ? 50.0f : 0.0f);
            exact += s;
            magnitude += s;
        }
        float whole = 0.0f;
        int splits = 0;
        for (uint64_t others = 0; others < 64; ++others) {  // ever larger batches around the job
            std::vector<Job> jobs{job(1000, spp)};
            if (others) jobs.push_back(job(250 * others, 300));
            uint32_t a, b;
            split_jobs(jobs, 1024, others > 0, a, b);
            const float v = pixel_sum(sample, jobs[0]);
            if (others == 0) whole = v;  // unsplit
            if (v != whole) ++errors;
            splits += jobs[0].units > 1;
        }
        if (std::fabs(whole - exact) > 6e-8 * spp * magnitude) ++errors;
        printf("%d samples: %d splits\n", spp, splits);
        if (spp >= 5 && (splits < 2 || (spp < 64 && splits == 63))) ++errors;
    }
    return errors;
}

int main() {
    const uint64_t lanes = 152 * kBatchLanes;
    const uint64_t view = 16384ull * 16384;
    std::vector<std::vector<Job>> lists = {
        {job(1, 1)},
        {job(300, 5), job(221, 33), job(15, 1)},
        {job(512 * 512, 60), job(957, 7), job(256, 2), job(64, 1), job(1, 9)},
        {job(64 * 64, 4096)},
        {job(view, 3)},
        std::vector<Job>(27, job(512 * 512, 48)),
    };
    // 4,293,771,840 pixels, all but a small job of many samples at one sample each.
    std::vector<Job> big(15, job(view, 1));
    big.push_back(job(16384ull * 16250, 1));
    big.push_back(job(1000 * 1000, 2000));
    lists.push_back(big);
    std::vector<Job> edge(15, job(view, 1));  // one sample each, up to the limit on pixels
    edge.push_back(job(view - 256, 1));
    lists.push_back(edge);
    int errors = check_sums();
    for (bool split : {false, true})
        for (std::vector<Job> jobs : lists) {
            uint32_t split_pixels, parts;
            const uint64_t items = split_jobs(jobs, lanes, split, split_pixels, parts);
            uint64_t next = 0, p = 0, d = 0;
            for (const Job& j : jobs) {
                if (j.item_begin != next) ++errors;
                next += (uint64_t)j.units * j.pixels;
                const uint64_t runs = ((uint64_t)j.spp + j.run_spp - 1) / j.run_spp;
                if (j.units != 1 && j.units != runs) ++errors;
                if (!split && j.units != 1) ++errors;
                if (j.units == 1) continue;
                if (j.part_begin != p || j.done_begin != d) ++errors;
                p += runs * j.pixels;
                d += j.pixels;
            }
            printf("%zu jobs: %llu items\n", jobs.size(), (unsigned long long)items);
            if (items != next || parts != p || split_pixels != d) ++errors;
            if (items > 0xFFFFFF00ull || (p && items > kMaxSplitItems) || p > kMaxStoredRuns) ++errors;
        }
    printf(errors ? "FAIL %d\n" : "OK\n", errors);
    return errors ? 1 : 0;
}
"""


def test_items_cover_every_sample_once_and_fit_32_bits(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip().endswith("OK"), out.stdout
