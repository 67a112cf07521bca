// FP64 Schur-complement update of a large front after a 256-column pivot
// panel (the FP64 counterpart of the tensor-core kernel in schur_tc.cu, same
// work lists and tile enumeration):
//     C(I, J) -= A_I * A_J'     128 x 128 tile, K <= 256 panel columns
// on the FP64 matrix instructions (dmma.cuh): a tile is four CTAs of 64 x 64
// (128 threads, warps of 32 x 32, three CTAs per SM, so one CTA's epilogue
// runs under the others' products), operand chunks of 16 panel columns
// through a three-stage cp.async ring.  The FP64 pipe is the busiest unit, 58 %
// of the longest launch of a 40^3 factor: 16.4 k cycles of it per CTA for 0.3 MB
// of operands and C; the rest is whole tiles at the fronts' edges, the last wave
// and the chunk loads.
// Measured on the 48^3 grid's FP64 factor (80 launches): 6.5 ms, 18 TFLOP/s
// with the launches' tails, against 14.1 ms for 128 x 128 tiles of register
// FMAs (an LDS.128 per four of them) and 7.8 ms for CTAs of 64 x 128 (two per
// SM, half as many to fill the chip's last wave).
#include <cuda_runtime.h>

#include <cstdint>

#include "device_common.cuh"
#include "dmma.cuh"
#include "kernels.hpp"

namespace mdgpu {

namespace f64k {
constexpr int BT = 128;  // the work lists' tile
constexpr int KC = 16, THREADS = 128, STAGES = 3;
constexpr int BM = 64, BN = 64, PIECES = (BT / BM) * (BT / BN);
constexpr int LDA = BM + 4, LDB = BN + 4;
constexpr int STAGE = KC * (LDA + LDB);  // doubles: A and B chunk
constexpr size_t SMEM_BYTES = (size_t)STAGES * STAGE * sizeof(double);
constexpr int MT = 2, NT = 2;  // a warp's 32 x 32
}  // namespace f64k

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// rows r0 .. r0 + R - 1 (zeros from row m on) of the panel columns [col, col +
// 16) that lie before kend, into dst (ld LD)
template <int R, int LD>
__device__ __forceinline__ void load_rows(double* dst, const double* panelp, int64_t ldl, int r0,
                                          int m, int col, int kend) {
    constexpr int PAIRS = R / 2, STEP = f64k::THREADS / PAIRS;
    const int r2 = (threadIdx.x % PAIRS) * 2, row = r0 + r2;
#pragma unroll
    for (int q = threadIdx.x / PAIRS; q < f64k::KC; q += STEP) {
        // rows beyond the front (or a partial pair) and columns beyond the
        // panel are zero-filled; the source address then stays in bounds
        const int bytes = (col + q < kend && row < m) ? min(2, m - row) * 8 : 0;
        cp_async16(dst + q * LD + r2, panelp + (bytes ? (int64_t)(col + q) * ldl + row : 0), bytes);
    }
}

__global__ void __launch_bounds__(f64k::THREADS, 3)
    k_schur_f64(const FrontDesc* __restrict__ fronts, const int* __restrict__ items,
                const int* __restrict__ before, int nitems, int panel, int PW,
                double* __restrict__ Ls, double* __restrict__ Us) {
    using namespace f64k;
    extern __shared__ __align__(16) double sm[];
    const int tile = blockIdx.x / PIECES, piece = blockIdx.x % PIECES;
    const int it = find_item(before, nitems, tile);
    const FrontDesc f = fronts[items[it]];
    const int k0 = panel * PW;
    const int K = min(PW, f.c - k0);
    const int cbeg = min(k0 + PW, f.c);
    int ii, jj;
    lower_index(tile - before[it], ii, jj);
    // this piece's first row and column
    const int R0 = (cbeg / BT + ii) * BT + (piece % (BT / BM)) * BM;
    const int C0 = (cbeg / BT + jj) * BT + (piece / (BT / BM)) * BN;
    // nothing below the diagonal, or past the front, or before the update's
    // first column
    if (C0 > R0 + BM - 1 || R0 >= f.m || C0 + BN <= cbeg) return;
    const double* panelp = Ls + f.loff;
    const int nchunks = (K + KC - 1) / KC;
    const int warp = threadIdx.x >> 5;
    const int wr = (warp & 1) * 32, wc = (warp >> 1) * (BN / 2);
    const bool active = C0 + wc <= R0 + wr + 31 && R0 + wr < f.m && C0 + wc + BN / 2 > cbeg;

    auto load_chunk = [&](int ch) {
        if (ch < nchunks) {
            double* As = sm + (ch % STAGES) * STAGE;
            load_rows<BM, LDA>(As, panelp, f.ldl, R0, f.m, k0 + ch * KC, k0 + K);
            load_rows<BN, LDB>(As + KC * LDA, panelp, f.ldl, C0, f.m, k0 + ch * KC, k0 + K);
        }
        cp_async_commit();
    };

    double acc[MT][NT][2][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[m][n][h][e] = 0.0;

    load_chunk(0);
    load_chunk(1);
    for (int ch = 0; ch < nchunks; ++ch) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();  // chunk ch landed for everyone; chunk ch - 1 is consumed
        load_chunk(ch + 2);
        const double* As = sm + (ch % STAGES) * STAGE;
        if (active)
            dmma_k16<MT, NT, LDA, LDB>(As + wr, As + KC * LDA + wc, acc);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!active) return;
    // epilogue, 16 columns at a time: a lane's 4 columns of two adjacent rows
    // per 16-row block, old values gathered first
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        double* p[MT][2][4];
        double old[MT][2][4];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int row = R0 + wr + 16 * m + 2 * g + r, col = C0 + wc + 16 * n + 4 * t + k;
                    const bool ok = row < f.m && col >= cbeg && row >= col;
                    p[m][r][k] = ok ? front_elem(Ls, Us, f, row, col) : nullptr;
                }
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int k = 0; k < 4; ++k) old[m][r][k] = p[m][r][k] ? *p[m][r][k] : 0.0;
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (p[m][r][k]) *p[m][r][k] = old[m][r][k] - acc[m][n][k & 1][2 * r + (k >> 1)];
    }
}

void init_schur_f64() {
    cudaFuncSetAttribute(k_schur_f64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)f64k::SMEM_BYTES);
}

void launch_schur_f64(const DevPlan& D, const WorkList& w, int panel, int PW, double* Ls,
                      double* Us, cudaStream_t st) {
    k_schur_f64<<<w.nctas * f64k::PIECES, f64k::THREADS, f64k::SMEM_BYTES, st>>>(
        D.fronts, D.psched.items + w.off, D.psched.before + w.off, w.nitems, panel, PW, Ls, Us);
}

}  // namespace mdgpu
