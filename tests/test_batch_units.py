"""How a batch's pixels are split into work items (csrc/batch_units.h), checked
on the host: a small C++ program splits job lists, small ones and ones whose
items outgrow 32 bits, and checks that every sample of every pixel belongs to
exactly one item."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "aqua-engine_gb300", "csrc")

PROGRAM = r"""
#include "batch_units.h"
#include <cstdio>

using namespace aq;

struct Job {
    int32_t spp;
    uint32_t pixels, item_begin, units, unit_spp, part_begin, done_begin;
};
static Job job(uint64_t pixels, int spp) {
    Job j{};
    j.pixels = (uint32_t)pixels;
    j.spp = spp;
    return j;
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
    };
    // 4,293,771,840 pixels, all but a small job of many samples at one sample each.
    std::vector<Job> big(15, job(view, 1));
    big.push_back(job(16384ull * 16250, 1));
    big.push_back(job(1000 * 1000, 2000));
    lists.push_back(big);
    std::vector<Job> edge(15, job(view, 1));  // one sample each, up to the limit on pixels
    edge.push_back(job(view - 256, 1));
    lists.push_back(edge);
    int errors = 0;
    for (bool split : {false, true})
        for (std::vector<Job> jobs : lists) {
            uint32_t split_pixels, parts;
            const uint64_t items = split_jobs(jobs, lanes, split, split_pixels, parts);
            uint64_t next = 0, p = 0, d = 0;
            for (const Job& j : jobs) {
                if (j.item_begin != next) ++errors;
                next += (uint64_t)j.units * j.pixels;
                if (j.unit_spp == 0 || (uint64_t)(j.units - 1) * j.unit_spp >= (uint64_t)j.spp ||
                    (uint64_t)j.units * j.unit_spp < (uint64_t)j.spp)
                    ++errors;
                if (!split && j.units != 1) ++errors;
                if (j.units == 1) continue;
                if (j.part_begin != p || j.done_begin != d) ++errors;
                p += (uint64_t)j.units * j.pixels;
                d += j.pixels;
            }
            printf("%zu jobs: %llu items\n", jobs.size(), (unsigned long long)items);
            if (items != next || parts != p || split_pixels != d) ++errors;
            if (items > 0xFFFFFF00ull) ++errors;
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
