// grouped.cuh -- device descriptors of the uneven (grouped) batched GEMM,
// shared by its three kernels: the mma.sync warp-grid kernel (grouped.cu),
// the tcgen05 ring kernel (h16_ring.cu, FP16 / BF16) and the FP64 ring kernel
// (f64_ring.cu).
#pragma once
#include <vector>

#include "kami_common.cuh"

namespace kami {

// One problem: shape, warp partition (mma.sync kernel), element offsets of
// A (M x K), B (N x K) and C (M x N) and their leading dimensions.
struct GroupedDesc
{
    int M, N, K, cfg;
    int64_t a_off, b_off, c_off;
    int lda, ldb, ldc;
};

struct GroupedParams
{
    const GroupedDesc *desc; // problems in schedule order
    const int *cta_begin;    // ctas + 1 offsets into desc
    const void *A;
    const void *B;
    void *C;
    int out_type;
    double alpha, beta;
    int num_iter;
    int small_begin, small_end; // desc range of problems run by single warps
};

// 16-bit ring kernel (h16_ring.cu): plans, and uniform batches
// (h16_ring_launch)
int h16_ring_smem();
int h16_ring_groups(int count, const int *M, const int *N); // problem lists of a CTA
void h16_ring_schedule(const std::vector<std::vector<int>> &lists, const int *M, const int *N, const int *K,
                       const int64_t *ao, const int64_t *bo, const int64_t *co, std::vector<char> *out,
                       std::vector<int> *begin, int groups);
int h16_ring_plan_launch(const GroupedParams &p, const void *chunks, bool bf16, int ctas, int groups, cudaStream_t s);
int h16_ring_launch(const GemmArgs &g, int in_type, cudaStream_t s);
int h16_ring_read_error(int *flag);

// FP64 ring kernel (f64_ring.cu): plans, and uniform batches (f64_ring_launch)
int f64_ring_smem();
size_t f64_ring_schedule(const std::vector<std::vector<int>> &lists, const int *M, const int *N, const int *K,
                         const int64_t *ao, const int64_t *bo, const int64_t *co, std::vector<char> *out,
                         std::vector<int> *begin);
int f64_ring_plan_launch(const GroupedParams &p, const void *chunks, int ctas, cudaStream_t s);
int f64_ring_launch(const GemmArgs &g, cudaStream_t s);
int f64_ring_read_error(int *flag);

} // namespace kami
