// The tensor-core kernels' waits run out (a limit of no polls at all): each kernel waits for what it has in flight,
// frees its TMEM and reports, and the calls after it give what they gave before.  Arguments: conv, or ctpt and
// the number of inputs.  Exit status 0 when all hold.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/shmoai_ckks.h"
#include "../../shmoai_b200/csrc/core.hpp"

struct shm_context {
    shm::Context *c;
};

static int bad = 0;
static void expect(const char *what, int got, int want) {
    if (got != want) std::printf("%s: %d, expected %d (%s)\n", what, got, want, shm_last_error()), bad++;
}
static constexpr uint32_t nq = 4, np = 2, N = 4096;

static shm_context *open() {
    shm_context *ctx = nullptr;
    const int bits[nq + np] = {50, 45, 45, 45, 50, 50};
    expect("create", shm_context_create(&ctx, 12, bits, nq, np, 0), SHM_OK);
    return ctx;
}
static uint64_t *words(shm_context *ctx, size_t n) {
    void *p = nullptr;
    expect("malloc", shm_malloc(ctx, n * 8, &p, nullptr), SHM_OK);
    return (uint64_t *)p;
}
static std::vector<uint64_t> download(shm_context *ctx, const uint64_t *p, size_t n, int want) {
    std::vector<uint64_t> h(n);
    expect("download", shm_memcpy(ctx, h.data(), p, n * 8, SHM_COPY_D2H, nullptr), want);
    return h;
}

// enough digits for several tiles of a CTA (two buffers in use)
static std::vector<uint64_t> keyswitch(bool give_up) {
    const uint32_t n = 320;
    shm_context *ctx = open();
    uint64_t *d = words(ctx, (size_t)n * nq * N), *key = words(ctx, 4ull * (nq + np) * N), *out = words(ctx, 2ull * n * nq * N);
    const size_t ws_bytes = shm_keyswitch_workspace_bytes(ctx, n, nq);
    uint64_t *ws = words(ctx, ws_bytes / 8);
    expect("sample", shm_sample_uniform(ctx, d, n, nq, 1, nullptr), SHM_OK);
    expect("sample", shm_sample_uniform(ctx, key, 4, nq + np, 2, nullptr), SHM_OK);
    if (give_up) ctx->c->wait_limit = 0;
    expect("keyswitch", shm_keyswitch(ctx, d, key, out, n, nq, ws, ws_bytes, nullptr), SHM_OK);
    expect("synchronize", shm_synchronize(ctx, nullptr), give_up ? SHM_ECUDA : SHM_OK);
    auto h = download(ctx, out, 2ull * n * nq * N, give_up ? SHM_ECUDA : SHM_OK);
    for (uint64_t *p : {d, key, out, ws}) expect("free", shm_free(ctx, p, nullptr), SHM_OK);
    shm_context_destroy(ctx);
    return h;
}

static void ctpt(uint32_t n_in) {
    const uint32_t n_out = 200, L = 3;
    shm_context *ctx = open();
    const size_t row = 2ull * L * N, ws_bytes = shm_ctpt_matmul_workspace_bytes(ctx, n_in, n_out, L);
    uint64_t *X = words(ctx, n_in * row), *Y = words(ctx, n_out * row), *W = words(ctx, (size_t)n_in * n_out);
    uint64_t *ws = words(ctx, ws_bytes / 8 + 1);
    std::vector<int64_t> w((size_t)n_in * n_out);
    for (size_t i = 0; i < w.size(); i++) w[i] = (int64_t)((i * 2654435761u) % 2000001u) - 1000000;
    expect("sample", shm_sample_uniform(ctx, X, 2 * n_in, L, 3, nullptr), SHM_OK);
    expect("upload", shm_memcpy(ctx, W, w.data(), w.size() * 8, SHM_COPY_H2D, nullptr), SHM_OK);
    std::vector<uint64_t> y[2];
    for (int turn = 0; turn < 3; turn++) {
        const bool give_up = turn == 1;
        ctx->c->wait_limit = give_up ? 0 : shm::kSpinLimit;
        expect("matmul", shm_ctpt_matmul(ctx, X, (int64_t *)W, Y, n_in, n_out, L, ws, ws_bytes, nullptr),
               give_up ? SHM_ECUDA : SHM_OK);
        if (!give_up) y[turn / 2] = download(ctx, Y, n_out * row, SHM_OK);
    }
    if (y[0] != y[1]) std::printf("results differ after a given-up wait\n"), bad++;
    for (uint64_t *p : {X, Y, W, ws}) expect("free", shm_free(ctx, p, nullptr), SHM_OK);
    shm_context_destroy(ctx);
}

int main(int argc, char **argv) {
    if (argc > 1 && !std::strcmp(argv[1], "conv")) {
        const auto a = keyswitch(false);
        keyswitch(true);
        if (keyswitch(false) != a) std::printf("results differ after a given-up wait\n"), bad++;
    } else if (argc > 2) {
        ctpt((uint32_t)std::atoi(argv[2]));
    } else {
        bad++;
    }
    std::printf(bad ? "FAIL\n" : "OK\n");
    return bad != 0;
}
