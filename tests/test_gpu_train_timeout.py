"""A training step whose kernel reports an expired wait leaves the network as it
was: weights, moments, average and both weight images, and the step count. The
flag is set from the host, as the kernel would have; the step after it is the
step that a network without the failure takes, bit for bit."""
from __future__ import annotations

import pytest

import native

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include "nrc.h"
using namespace aq;

static const size_t nrc_tc_bytes = 5 * kNrcTcLayerBytes + kNrcTcOutRows * 64 * 2;

struct State {
    std::vector<uint8_t> data;
    int64_t step;
};
// Weights, moments, gradient, average and the two tcgen05 weight images.
static bool state_of(const aqua_nrc* n, State& s) {
    const NrcNet& t = n->net;
    s.step = t.step;
    s.data.clear();
    auto add = [&](const void* p, size_t bytes) {
        const size_t at = s.data.size();
        s.data.resize(at + bytes);
        return cudaMemcpy(&s.data[at], p, bytes, cudaMemcpyDeviceToHost) == cudaSuccess;
    };
    for (const float* p : {t.w, t.m, t.v, t.grad, t.ema})
        if (!add(p, 4 * kNrcParams)) return false;
    return add(t.img_tc, nrc_tc_bytes) && add(t.img_tc_w, nrc_tc_bytes);
}

int main() {
    aqua_ctx* ctx = nullptr;
    aqua_nrc *a = nullptr, *b = nullptr;
    CHECK(aqua_create(&ctx, nullptr) == AQUA_OK);
    aqua_nrc_cfg cfg;
    aqua_nrc_defaults(&cfg);
    cfg.ema_decay = 0.9f;
    CHECK(aqua_nrc_create(ctx, &cfg, &a) == AQUA_OK && aqua_nrc_create(ctx, &cfg, &b) == AQUA_OK);
    const int rows = 300;
    std::vector<uint16_t> x(64 * rows);
    std::vector<float> t(3 * rows);
    uint32_t r = 1;
    for (auto& v : x) v = (uint16_t)(0x3c00u + ((r = r * 1664525u + 1013904223u) >> 25));  // small positive bf16
    for (auto& v : t) v = (float)((r = r * 1664525u + 1013904223u) >> 8) / 16777216.0f;
    double la = 0.0, lb = 0.0;
    auto step = [&](aqua_nrc* n, double& l) { return aqua_nrc_train_step(ctx, n, x.data(), t.data(), rows, &l, 0); };
    State before, after, plain;
    for (int round = 0; round < 3; ++round) {  // the first step, and later ones
        CHECK(state_of(a, before));
        const uint32_t one = 1;
        CHECK(cudaMemcpy(a->net.tc_err, &one, 4, cudaMemcpyHostToDevice) == cudaSuccess);
        CHECK(step(a, la) == AQUA_ERR_TIMEOUT);
        CHECK(state_of(a, after));
        CHECK(after.step == before.step);
        CHECK(after.data == before.data);
        CHECK(step(a, la) == AQUA_OK && step(b, lb) == AQUA_OK);
        CHECK(la == lb);
        CHECK(state_of(a, after) && state_of(b, plain));
        CHECK(after.step == plain.step && after.data == plain.data);
        CHECK(after.data != before.data);
    }
    // New weights start over.
    std::vector<float> w(kNrcParams);
    CHECK(aqua_nrc_get_weights(ctx, b, w.data()) == AQUA_OK);
    CHECK(aqua_nrc_set_weights(ctx, a, w.data()) == AQUA_OK && a->net.step == 0);
    const uint32_t one = 1;
    CHECK(cudaMemcpy(a->net.tc_err, &one, 4, cudaMemcpyHostToDevice) == cudaSuccess);
    CHECK(step(a, la) == AQUA_ERR_TIMEOUT && a->net.step == 0);
    CHECK(step(a, la) == AQUA_OK && a->net.step == 1);
    aqua_nrc_destroy(ctx, a);
    aqua_nrc_destroy(ctx, b);
    aqua_destroy(ctx);
    printf("OK\n");
    return 0;
}
"""


def test_a_timed_out_step_changes_nothing(tmp_path):
    native.run(tmp_path, PROGRAM)
