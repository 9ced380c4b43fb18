// Host paths of the library against the fake CUDA runtime; `name` on the
// command line picks one.  Prints "ok" or the first condition that failed.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>
#include "../pagani-toolkit_b200/csrc/pg_internal.cuh"
#include "../pagani-toolkit_b200/csrc/tune.cuh"
#include "fake_cudart.h"

#define CHECK(x)                                            \
    do {                                                    \
        if (!(x)) {                                         \
            printf("line %d: %s\n", __LINE__, #x);          \
            return 1;                                       \
        }                                                   \
    } while (0)

// a copy of one thread fails: the others' may be on their way into the staging
// buffers, which the next call uses again
static int large_copy_that_fails(pg_ctx* ctx)
{
    if (std::thread::hardware_concurrency() < 4) return 0;   // one thread then copies everything directly
    const size_t bytes = 40u << 20;
    std::vector<unsigned char> src(bytes), dst(bytes);
    for (size_t k = 0; k < bytes; k++) src[k] = (unsigned char)(k * 2654435761u >> 13);
    for (int at : {0, 1, 5, 13, 19}) {
        fake::copies = 0;
        fake::fail_copy = at;
        CHECK(pg_d2h_large(ctx, dst.data(), src.data(), bytes) == PG_ERR_CUDA);
        CHECK(fake::open_copies == 0);
        fake::fail_copy = -1;
        CHECK(pg_d2h_large(ctx, dst.data(), src.data(), bytes) == PG_OK);
        CHECK(dst == src);
    }
    return 0;
}

// scratch that no call uses goes when memory is short, and only then
static int idle_buffers_make_room(pg_ctx* ctx)
{
    void *a, *b, *c;
    fake::device_limit = 1000;
    CHECK(pg_ws(ctx, "a", 400, &a) == PG_OK);
    CHECK(pg_ws(ctx, "b", 400, &b) == PG_OK);
    CHECK(pg_ws(ctx, "c", 400, &c) == PG_ERR_NOMEM);      // both are in use
    pg_ws_idle(ctx, "a");
    CHECK(pg_ws(ctx, "a", 400, &c) == PG_OK && c == a);   // taken again: the same buffer, in use
    CHECK(pg_ws(ctx, "c", 400, &c) == PG_ERR_NOMEM);
    pg_ws_idle(ctx, "a");
    CHECK(pg_ws(ctx, "c", 400, &c) == PG_OK);
    CHECK(fake::device_bytes == 2 * 450);
    CHECK(ctx->ws["a"].p == nullptr && ctx->ws["b"].p == b);
    // graphs too
    pg_ws_idle(ctx, "b");
    const int32_t R[3] = {0, 1, 2}, C[2] = {1, 0};
    pg_graph* g = nullptr;
    fake::device_limit = 905;
    CHECK(pg_graph_from_csr(ctx, R, C, nullptr, 2, 2, 0, &g) == PG_OK);
    CHECK(ctx->ws["b"].p == nullptr && ctx->ws["c"].p == c);
    CHECK(pg_graph_free(g) == PG_OK);
    CHECK(fake::device_bytes == 450);
    return 0;
}

// no pinned memory for the staging buffers: the plain copy
static int large_copy_without_staging(pg_ctx* ctx)
{
    const size_t bytes = 20u << 20;
    std::vector<unsigned char> src(bytes, 7), dst(bytes, 0);
    fake::host_limit = 1 << 20;
    CHECK(pg_d2h_large(ctx, dst.data(), src.data(), bytes) == PG_OK);
    CHECK(dst == src && fake::copies == 1);
    return 0;
}

// a tuning file from another build: its choice is not among the candidates
static int saved_choice_that_does_not_fit(pg_ctx* ctx)
{
    const char* path = getenv("PAGANI_TUNE_CACHE");
    CHECK(path);
    const std::string key = tune_key("test", 1000, 8000), other = tune_key("test", 100000, 800000);
    FILE* f = fopen(path, "w");
    CHECK(f);
    fprintf(f, "%s 4 4 0.1\n%s 8 2 0.1\n", key.c_str(), other.c_str());
    fclose(f);
    const std::vector<TuneChoice> cands = {{4, 2}, {8, 2}};
    TuneChoice best{0, 0};
    int runs = 0;
    auto run = [&](const TuneChoice&) -> pg_status { runs++; return PG_OK; };
    CHECK(tune_pick(ctx, other, cands, &best, run) == PG_OK && best.a == 8 && best.b == 2 && runs == 0);
    CHECK(tune_pick(ctx, key, cands, &best, run) == PG_OK && best.b == 2 && runs == 4);
    return 0;
}

// the error of a call that failed is not taken for the next call's launch error
static int error_that_is_over(pg_ctx* ctx)
{
    char a[8] = {}, b[8] = {};
    fake::fail_copy = 0;
    CHECK(pg_d2h(ctx, a, b, sizeof a) == PG_ERR_CUDA);
    fake::fail_copy = -1;
    int32_t cnt[3] = {1, 1, 0}, R[3] = {};
    CHECK(pg_row_offsets(ctx, cnt, 2, R) == PG_OK);   // two launches, each checked
    return 0;
}

int main(int argc, char** argv)
{
    pg_ctx* ctx;
    if (argc < 2 || pg_create(&ctx, 0) != PG_OK) return 2;
    int rc = 2;
    if (!strcmp(argv[1], "large_copy_that_fails")) rc = large_copy_that_fails(ctx);
    if (!strcmp(argv[1], "idle_buffers_make_room")) rc = idle_buffers_make_room(ctx);
    if (!strcmp(argv[1], "large_copy_without_staging")) rc = large_copy_without_staging(ctx);
    if (!strcmp(argv[1], "saved_choice_that_does_not_fit")) rc = saved_choice_that_does_not_fit(ctx);
    if (!strcmp(argv[1], "error_that_is_over")) rc = error_that_is_over(ctx);
    pg_destroy(ctx);
    if (rc == 0) puts("ok");
    return rc;
}
