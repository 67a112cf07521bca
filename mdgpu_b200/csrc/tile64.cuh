// 64 x 64 FP64 products of operands gathered element by element from global
// memory, over a CTA of 128 threads (four warps of 32 x 32 outputs on the
// matrix instructions, dmma.cuh): K in stages of 32, double-buffered 8-byte
// cp.async into K-slowest blocks of leading dimension 68 (or 64 x 16 products,
// warps of 16 x 16, for operands of at most 16 columns).  The gathers take
// operands of any store, alignment and symmetry; their index arithmetic (16
// elements of each operand per thread and stage) stays under the stage's 2 k
// cycles of products.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "dmma.cuh"

namespace mdgpu {

namespace t64 {
constexpr int T = 64, KS = 32, LD = T + 4, THREADS = 128;
constexpr int BLOCK = KS * LD;                   // doubles of one operand's stage
constexpr size_t SMEM_BYTES = 4 * BLOCK * sizeof(double);
using Acc = double[2][2][2][4];

template <int MT, int NT>
__device__ __forceinline__ void zero(double (&acc)[MT][NT][2][4]) {
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[m][n][h][e] = 0.0;
}
// the columns of B that an accumulator's shape takes, a warp's first row and
// column
template <int MT>
constexpr int cols() {
    return MT == 2 ? T : 16;
}
template <int MT>
__device__ __forceinline__ int row0() {
    const int warp = threadIdx.x >> 5;
    return MT == 2 ? (warp & 1) * 32 : warp * 16;
}
template <int MT>
__device__ __forceinline__ int col0() {
    return MT == 2 ? (threadIdx.x >> 6) * 32 : 0;
}
// f(row, column, value) over this thread's outputs
template <int MT, int NT, typename F>
__device__ __forceinline__ void each(const double (&acc)[MT][NT][2][4], F&& f) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int r = 0; r < 2; ++r)
                    f(row0<MT>() + 16 * m + 2 * g + r, col0<MT>() + 16 * n + 4 * t + k,
                      acc[m][n][k & 1][2 * r + (k >> 1)]);
}
// acc += A B' over 16 steps of two K-slowest blocks
template <int MT, int NT>
__device__ __forceinline__ void step16(const double* As, const double* Bs,
                                       double (&acc)[MT][NT][2][4]) {
    dmma_k16<MT, NT, LD, LD>(As + row0<MT>(), Bs + col0<MT>(), acc);
}
// one operand stage: dst[k * LD + x] = *at(k0 + k, x), zero where at() gives
// null; KFAST: neighbouring threads take neighbouring k (operands contiguous
// along k), else neighbouring x
template <bool KFAST, int NX, typename F>
__device__ __forceinline__ void load(double* dst, int k0, F&& at) {
#pragma unroll 4
    for (int idx = threadIdx.x; idx < KS * NX; idx += THREADS) {
        const int k = KFAST ? idx & (KS - 1) : idx / NX, x = KFAST ? idx / KS : idx & (NX - 1);
        const double* p = at(k0 + k, x);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(dst + k * LD + x))),
                     "l"(__cvta_generic_to_global(p ? p : at.any)), "r"(p ? 8 : 0)
                     : "memory");
    }
}
// An operand: fn(k, x) -> pointer or null; any: a valid address for the zeros
template <typename F>
struct Op {
    const double* any;
    F fn;
    __device__ __forceinline__ const double* operator()(int k, int x) const { return fn(k, x); }
};
template <typename F>
__device__ __forceinline__ Op<F> op(const double* any, F fn) {
    return Op<F>{any, fn};
}
// acc += sum over k in [k0, k1) of A(k, row) B(k, column); sm: SMEM_BYTES.
// Ends with a CTA barrier (sm and what the operands read may be reused).
template <bool AK, bool BK, typename FA, typename FB, int MT, int NT>
__device__ __forceinline__ void product(double* sm, int k0, int k1, const FA& a, const FB& b,
                                        double (&acc)[MT][NT][2][4]) {
    auto issue = [&](int k, int slot) {
        if (k < k1) {
            load<AK, T>(sm + slot * 2 * BLOCK, k, a);
            load<BK, cols<MT>()>(sm + slot * 2 * BLOCK + BLOCK, k, b);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    issue(k0, 0);
    int slot = 0;
    for (int k = k0; k < k1; k += KS, slot ^= 1) {
        issue(k + KS, slot ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const double* As = sm + slot * 2 * BLOCK;
        step16(As, As + BLOCK, acc);
        if (k + 16 < k1) step16(As + 16 * LD, As + BLOCK + 16 * LD, acc);
        __syncthreads();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}
}  // namespace t64

}  // namespace mdgpu
