// Host paths of the library against the fake CUDA runtime; `name` on the
// command line picks one.  Prints "ok" or the first condition that failed.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>
#include "../pagani-toolkit_b200/csrc/pg_internal.cuh"
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

int main(int argc, char** argv)
{
    pg_ctx* ctx;
    if (argc < 2 || pg_create(&ctx, 0) != PG_OK) return 2;
    int rc = 2;
    if (!strcmp(argv[1], "large_copy_that_fails")) rc = large_copy_that_fails(ctx);
    pg_destroy(ctx);
    if (rc == 0) puts("ok");
    return rc;
}
