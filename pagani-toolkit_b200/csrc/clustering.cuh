// clustering.cuh -- clustering pieces that the surrogate pipeline (runner.cu)
// and the batched FW tool enqueue without host round trips.
#pragma once
#include "pg_internal.cuh"

struct BinaryCpArgs {
    unsigned long long* tri2;   // per node: twice the triangle count
    int* counter;               // dynamic node scheduler
    size_t smem;                // neighbour bitmap bytes
};
// Sizes the workspace and sets the kernel's shared-memory limit.
pg_status binary_cp_prepare(pg_ctx* ctx, int n, BinaryCpArgs* a);
// Enqueues Cp (U/Cp/Cp/Cp.cpp:21-116) of (R, C): cp float[n], exact
// triangles (tri, optional), FP64 mean over all n nodes -- device pointers.
pg_status binary_cp_enqueue(pg_ctx* ctx, const BinaryCpArgs* a, const int32_t* R, const int32_t* C, int n, float* cp,
                            long long* tri, double* mean);

// Device state of one Onnela computation, cleared when it is enqueued.
struct OnnelaState {
    unsigned vmax;              // weight maximum (order-preserving bits)
    int general;                // the weights or rows need the general kernel
    int next;                   // dynamic node scheduler
};

struct OnnelaArgs {
    const int32_t *R, *C;
    const float* V;
    int n;
    int64_t nnz, vmax_entries;
    OnnelaState* state;
    double* roots = nullptr;    // per entry: cube root of the normalised weight
    int32_t* up = nullptr;      // per row: first entry above the row's own index
    size_t smem, smem_general;
    bool fast;                  // the neighbour table fits shared memory
    float* cp;
    double* mean;
};
// Sizes the workspace and sets the kernels' shared-memory limits; the graph's
// device arrays must stay where they are while the arguments are used.
pg_status onnela_prepare(pg_ctx* ctx, const pg_graph* g, int first_n, float* cp_dev, double* mean_dev, OnnelaArgs* a);
// Enqueues Onnela clustering (W/Cp/Cp/Cp_2.cpp:23-130): cp float[n] and the
// FP64 mean over all nodes -- device pointers.
pg_status onnela_enqueue(pg_ctx* ctx, const OnnelaArgs* a);
