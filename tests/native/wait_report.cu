// A kernel's given-up wait (here: the flag it would set, set from the host) reaches every call that hands out or
// builds on results, leaves memory and graphs releasable, and stays with its context.  Exit status 0 when all hold.
#include <cstdio>
#include <cstring>

#include "../../include/shmoai_ckks.h"
#include "../../shmoai_b200/csrc/core.hpp"

struct shm_context {
    shm::Context *c;
};

static int bad = 0;
static void expect(const char *what, int got, int want) {
    if (got != want) std::printf("%s: %d, expected %d (%s)\n", what, got, want, shm_last_error()), bad++;
}

struct Ks {  // a key switch's buffers
    shm_context *ctx = nullptr;
    void *d = nullptr, *key = nullptr, *out = nullptr, *ws = nullptr;
    size_t ws_bytes = 0;
    static constexpr uint32_t nq = 4, np = 2, N = 4096;
    void open() {
        const int bits[nq + np] = {50, 45, 45, 45, 50, 50};
        expect("create", shm_context_create(&ctx, 12, bits, nq, np, 0), SHM_OK);
        ws_bytes = shm_keyswitch_workspace_bytes(ctx, 1, nq);
        expect("malloc", shm_malloc(ctx, nq * N * 8, &d, nullptr), SHM_OK);
        expect("malloc", shm_malloc(ctx, 2 * 2 * (nq + np) * N * 8, &key, nullptr), SHM_OK);
        expect("malloc", shm_malloc(ctx, 2 * nq * N * 8, &out, nullptr), SHM_OK);
        expect("malloc", shm_malloc(ctx, ws_bytes, &ws, nullptr), SHM_OK);
        expect("sample", shm_sample_uniform(ctx, (uint64_t *)d, 1, nq, 1, nullptr), SHM_OK);
        expect("sample", shm_sample_uniform(ctx, (uint64_t *)key, 4, nq + np, 2, nullptr), SHM_OK);
        expect("synchronize", shm_synchronize(ctx, nullptr), SHM_OK);
    }
    int run(void *st) {
        return shm_keyswitch(ctx, (const uint64_t *)d, (const uint64_t *)key, (uint64_t *)out, 1, nq, ws, ws_bytes, st);
    }
    void close() {
        for (void *p : {d, key, out, ws}) expect("free", shm_free(ctx, p, nullptr), SHM_OK);
        shm_context_destroy(ctx);
    }
};

int main() {
    Ks a;
    a.open();
    void *st = nullptr;
    shm_graph *g = nullptr;
    expect("stream", shm_stream_create(a.ctx, &st), SHM_OK);
    expect("keyswitch", a.run(st), SHM_OK);
    expect("begin", shm_graph_begin(a.ctx, st), SHM_OK);
    expect("captured keyswitch", a.run(st), SHM_OK);
    expect("end", shm_graph_end(a.ctx, st, &g), SHM_OK);
    expect("launch", shm_graph_launch(g, st), SHM_OK);
    expect("synchronize", shm_synchronize(a.ctx, st), SHM_OK);

    *a.ctx->c->fault = 1;
    uint64_t word = 0;
    expect("synchronize after", shm_synchronize(a.ctx, st), SHM_ECUDA);
    if (!std::strstr(shm_last_error(), "gave up a wait")) std::printf("message: %s\n", shm_last_error()), bad++;
    expect("download after", shm_memcpy(a.ctx, &word, a.out, 8, SHM_COPY_D2H, st), SHM_ECUDA);
    expect("copy after", shm_memcpy(a.ctx, a.out, a.d, 8, SHM_COPY_D2D, st), SHM_ECUDA);
    expect("replay after", shm_graph_launch(g, st), SHM_ECUDA);
    expect("keyswitch after", a.run(st), SHM_ECUDA);
    expect("transform after", shm_ntt_forward(a.ctx, (uint64_t *)a.d, 1, Ks::nq, st), SHM_ECUDA);

    Ks b;  // another context is not concerned
    b.open();
    expect("other keyswitch", b.run(nullptr), SHM_OK);
    expect("other download", shm_memcpy(b.ctx, &word, b.out, 8, SHM_COPY_D2H, nullptr), SHM_OK);
    b.close();

    expect("stream release", shm_stream_destroy(a.ctx, st), SHM_OK);
    a.close();
    shm_graph_destroy(g);  // outlives its context's memory, not the flag
    std::printf(bad ? "FAIL\n" : "OK\n");
    return bad != 0;
}
