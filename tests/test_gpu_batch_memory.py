"""A batch that finds no room for its stored runs keeps whole pixels, with the
same image bit for bit, and is split again as soon as there is room."""
from __future__ import annotations

import pytest

import native

pytestmark = pytest.mark.gpu

PROGRAM = r"""
int main() {
    aqua_ctx* ctx = nullptr;
    aqua_scene* scene = nullptr;
    CHECK(aqua_create(&ctx, nullptr) == AQUA_OK);
    CHECK(aqua_make_procedural_scene(ctx, 2, 0, 64, 48, &scene) == AQUA_OK);
    const size_t n = 3 * 64 * 48;
    float* film = nullptr;
    CHECK(cudaMalloc(&film, 4 * n) == cudaSuccess);
    std::vector<float> split(n), whole(n), again(n);
    aqua_job job{};
    job.scene = scene;
    job.width = 64;
    job.height = 48;
    job.spp = 9;
    job.max_depth = 5;
    job.seed = 3;
    job.rgb_out = film;
    auto render = [&](std::vector<float>& out) {
        return cudaMemset(film, 0xff, 4 * n) == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess &&
               aqua_render_batch(ctx, &job, 1, nullptr, nullptr) == AQUA_OK &&
               cudaMemcpy(out.data(), film, 4 * n, cudaMemcpyDeviceToHost) == cudaSuccess;
    };
    CHECK(render(split));
    CHECK(ctx->batch.split_pixels == 64 * 48);
    // Another batch in between, then the first one short of memory.
    job.seed = 4;
    CHECK(render(again));
    job.seed = 3;
    fail_next_alloc(ctx);
    CHECK(render(whole));
    CHECK(ctx->batch.split_pixels == 0);
    CHECK(memcmp(whole.data(), split.data(), 4 * n) == 0);
    // The failure was a passing one.
    CHECK(render(again));
    CHECK(ctx->batch.split_pixels == 64 * 48);
    CHECK(memcmp(again.data(), split.data(), 4 * n) == 0);
    // A persistent render of the same view keeps whole pixels; the batch after it does not.
    for (int spp : {1, 9}) {
        aqua_integrator_cfg cfg;
        aqua_integrator_defaults(&cfg);
        cfg.spp = job.spp = spp;
        cfg.max_depth = 5;
        cfg.seed = 3;
        aqua_tuning t;
        aqua_tuning_defaults(&t);
        t.kernel = AQUA_KERNEL_PERSISTENT;
        t.use_graph = 1;
        CHECK(aqua_render(ctx, scene, &cfg, &t, film, AQUA_RENDER_DEVICE_FILM, nullptr) == AQUA_OK);
        CHECK(ctx->batch.split_pixels == 0);
        CHECK(render(again));
        CHECK(ctx->batch.split_pixels == (spp > 1 ? 64 * 48 : 0));
    }
    CHECK(memcmp(again.data(), split.data(), 4 * n) == 0);
    aqua_scene_free(ctx, scene);
    aqua_destroy(ctx);
    cudaFree(film);
    printf("OK\n");
    return 0;
}
"""


def test_a_batch_short_of_memory_is_whole_until_there_is_room(tmp_path):
    native.run(tmp_path, PROGRAM)
