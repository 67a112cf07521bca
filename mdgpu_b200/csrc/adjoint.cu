// Reverse mode of the multifrontal Cholesky factorization (FP64): from the
// gradient Lbar of a loss with respect to the entries of L (on L's pattern)
// to the gradient Abar with respect to the caller's lower-triangle values.
//
// The factor (the forward structure of Factor, mdgpu.cu:1394-1608) per front
// s with pivot block K (c columns) and update rows R (u rows):
//     F     = A_s + sum over children of extend(U_child)
//     L11   = chol(F11),   L21 = F21 L11^-T,   U = F22 - L21 L21'
// Reversed front by front from the root (all gradients with respect to the
// stored lower entries; an off-diagonal entry stands for both triangles):
//     Ubar  = Fbar of the parent on this front's update rows (the transpose
//             of the extend-add: a gather through the relative map)
//     L21bar -= (Ubar + Ubar') L21
//     F21bar  = L21bar L11^-1
//     L11bar -= tril(F21bar' L21)
//     F11bar  = the Cholesky adjoint of L11 (Murray 2016):
//               P = Phi(L11' L11bar), S = L11^-T P L11^-1,
//               F11bar = tril(S + S') with the diagonal of S
//     F22bar  = Ubar
// and Abar is Fbar at the positions where the front assembly put A's
// entries.  Only L and the gradients flowing down the tree are needed: the
// update matrices are neither stored for the reverse sweep nor recomputed.
//
// Fbar's pivot columns live in a store laid out like the L panels (it starts
// as Lbar, scattered there, and is turned into Fbar in place), Ubar in a
// store with the selected inverse's lifetimes (plan zuoff).
//
// Small fronts: one CTA per front and level.  Large fronts: 64 x 64 tiles of
// FP64 matrix-instruction products (tile64.cuh), the triangular solves by the
// stored inverses W_k of the diagonal tiles, in two classes per level:
//   narrow (c <= 64, one pivot tile; most levels of a tree have only these):
//     k_adj_rows   CTA per 64 update rows: L21bar - (Ubar + Ubar') L21 summed
//                  over all of u, times W, written, and the tile's part of
//                  F21bar' L21 kept
//     k_adj_pivot  CTA per front: the parts added, P, S, F11bar
//   wide (c > 64): one launch per step above, CTA per tile or, for the
//     solves, per 64 rows or columns (a chain of pivot tiles inside the CTA).
// Both are bound by latency (a level's few tiles leave most SMs idle, 128
// levels on a nested-dissection tree).  19 x 20 x 21 grid: 6.0 ms, against
// 117 ms for a CTA per front with scalar loops over global memory (72 ms of it
// the root's 552 columns).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device_common.cuh"
#include "kernels.hpp"
#include "tile64.cuh"

namespace mdgpu {

// Lbar (CSC of L: column j holds rows j.. in ascending order, diagonal
// first) into the panel store: panel (r, jj) of front s is entry
// Lp[first + jj] + r - jj for r >= jj; zero above the diagonal.  A warp per
// column, gridDim.y CTAs per front of the list (one CTA per front spent 0.4 ms
// on a root of 552 columns).
__global__ void __launch_bounds__(256)
    k_adj_scatter(const FrontDesc* __restrict__ fronts, const int* __restrict__ list,
                  const int64_t* __restrict__ Lp, const double* __restrict__ Lbar,
                  double* __restrict__ Fb) {
    const FrontDesc f = fronts[list[blockIdx.x]];
    const int lane = threadIdx.x & 31, nw = (blockDim.x >> 5) * gridDim.y;
    for (int jj = (threadIdx.x >> 5) + blockIdx.y * (blockDim.x >> 5); jj < f.c; jj += nw) {
        const double* src = Lbar + Lp[f.first_col + jj] - jj;
        double* col = Fb + f.loff + (int64_t)jj * f.ldl;
#pragma unroll 4
        for (int r = lane; r < f.m; r += 32) col[r] = r >= jj ? src[r] : 0.0;
    }
}

// odd: 1 if one of Lbar's values is infinite or a NaN (cleared by the caller).  A
// pass of its own at the rate of the memory; beside the scatter's stores the test
// took 0.1 ms on a 32^3 grid.
__global__ void __launch_bounds__(256)
    k_adj_check(int64_t lnz, const double* __restrict__ Lbar, int* __restrict__ odd) {
    const int64_t nt = (int64_t)gridDim.x * blockDim.x;
    int top = 0;  // the largest exponent
#pragma unroll 4
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < lnz; e += nt)
        top = max(top, __double2hiint(Lbar[e]) & 0x7fffffff);
    if (top >= 0x7ff00000) *odd = 1;
}

// Ubar of front s = Fbar of its parent on s's update rows (lower part): CTA
// per 16 columns, two per warp
__global__ void __launch_bounds__(256)
    k_adj_gather(const FrontDesc* __restrict__ fronts, const int* __restrict__ items,
                 const int* __restrict__ before, int nitems, const int* __restrict__ relmap,
                 const double* __restrict__ Fb, double* __restrict__ Fu,
                 const int64_t* __restrict__ zuoff) {
    const int it = find_item(before, nitems, blockIdx.x);
    const int s = items[it], blk = blockIdx.x - before[it];
    const FrontDesc f = fronts[s];
    const FrontDesc p = fronts[f.parent];
    const int u = f.m - f.c, lane = threadIdx.x & 31;
    const int64_t zf = zuoff[s], zp = zuoff[f.parent];
    const int* rm = relmap + f.rows_off + f.c;
    for (int b = 16 * blk + (threadIdx.x >> 5); b < min(16 * blk + 16, u); b += 8) {
        const int pb = rm[b];
        // the parent's column, by front row
        const double* src = pb < p.c ? Fb + p.loff + (int64_t)pb * p.ldl
                                     : Fu + zp - p.c + (int64_t)(pb - p.c) * p.ldu;
        double* dst = Fu + zf + (int64_t)b * f.ldu;
        for (int a0 = b + lane; a0 < u; a0 += 4 * 32) {
            double v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = a0 + 32 * k < u ? src[rm[a0 + 32 * k]] : 0.0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (a0 + 32 * k < u) dst[a0 + 32 * k] = v[k];
        }
    }
}

// One front by one CTA, scalar sums over the entries that L has: Lbar (pivot
// columns of Fb, rows 0..m) -> Fbar in place, with Ubar from Fu; W: c x c scratch.
__device__ void adj_front(int s, const FrontDesc* __restrict__ fronts,
                          const double* __restrict__ Ls, double* __restrict__ Fb,
                          const double* __restrict__ Fu, const int64_t* __restrict__ zuoff,
                          double* __restrict__ Wscr, const int64_t* __restrict__ woff) {
    const FrontDesc f = fronts[s];
    const int m = f.m, c = f.c, u = m - c;
    const int tid = threadIdx.x, nt = blockDim.x;
    const double* L = Ls + f.loff;  // L(r, k) = L[r + k ldl]
    double* G = Fb + f.loff;        // Lbar -> Fbar, same layout
    const int64_t zf = (f.parent >= 0 && u > 0) ? zuoff[s] : -1;
    double* W = Wscr + woff[s];     // c x c, column-major
    auto ubar = [&](int a, int b) -> double {  // (Ubar + Ubar')(a, b)
        if (a == b) return 2.0 * Fu[zf + a + (int64_t)a * f.ldu];
        const int hi = a > b ? a : b, lo = a > b ? b : a;
        return Fu[zf + hi + (int64_t)lo * f.ldu];
    };
    if (u > 0) {
        // L21bar -= (Ubar + Ubar') L21: outputs (a, k) (each reads L21 and
        // Ubar only)
        if (zf >= 0) {
            for (int64_t e = tid; e < (int64_t)u * c; e += nt) {
                const int a = (int)(e % u), k = (int)(e / u);
                double v = 0.0;
                for (int b = 0; b < u; ++b) v += ubar(a, b) * L[c + b + (int64_t)k * f.ldl];
                G[c + a + (int64_t)k * f.ldl] -= v;
            }
            __syncthreads();
        }
        // F21bar = L21bar L11^-1: row a solves x L11 = l, columns from last
        for (int a = tid; a < u; a += nt) {
            double* x = G + c + a;
            for (int k = c - 1; k >= 0; --k) {
                double v = x[(int64_t)k * f.ldl];
                for (int j = k + 1; j < c; ++j) v -= x[(int64_t)j * f.ldl] * L[j + (int64_t)k * f.ldl];
                x[(int64_t)k * f.ldl] = v / L[k + (int64_t)k * f.ldl];
            }
        }
        __syncthreads();
        // L11bar -= tril(F21bar' L21)
        for (int64_t e = tid; e < (int64_t)c * c; e += nt) {
            const int i = (int)(e % c), j = (int)(e / c);
            if (i < j) continue;
            double v = 0.0;
            for (int a = 0; a < u; ++a)
                v += G[c + a + (int64_t)i * f.ldl] * L[c + a + (int64_t)j * f.ldl];
            W[i + (int64_t)j * c] = v;
        }
        __syncthreads();
        for (int64_t e = tid; e < (int64_t)c * c; e += nt) {
            const int i = (int)(e % c), j = (int)(e / c);
            if (i >= j) G[i + (int64_t)j * f.ldl] -= W[i + (int64_t)j * c];
        }
        __syncthreads();
    }
    // Cholesky adjoint of the pivot block.  P = Phi(L11' L11bar) into W
    // (lower; P(i, j) = sum over k >= i of L(k, i) Lbar(k, j), diagonal halved)
    for (int64_t e = tid; e < (int64_t)c * c; e += nt) {
        const int i = (int)(e % c), j = (int)(e / c);
        double v = 0.0;
        if (i >= j) {
            for (int k = i; k < c; ++k) v += L[k + (int64_t)i * f.ldl] * G[k + (int64_t)j * f.ldl];
            if (i == j) v *= 0.5;
        }
        W[i + (int64_t)j * c] = v;
    }
    __syncthreads();
    // X = P L^-1: row i solves x L = p (columns from last), in place
    for (int i = tid; i < c; i += nt) {
        for (int k = c - 1; k >= 0; --k) {
            double v = W[i + (int64_t)k * c];
            for (int j = k + 1; j < c; ++j) v -= W[i + (int64_t)j * c] * L[j + (int64_t)k * f.ldl];
            W[i + (int64_t)k * c] = v / L[k + (int64_t)k * f.ldl];
        }
    }
    __syncthreads();
    // S = L^-T X: column j solves L' s = x (rows from last), in place
    for (int j = tid; j < c; j += nt) {
        double* sc = W + (int64_t)j * c;
        for (int k = c - 1; k >= 0; --k) {
            double v = sc[k];
            for (int r = k + 1; r < c; ++r) v -= L[r + (int64_t)k * f.ldl] * sc[r];
            sc[k] = v / L[k + (int64_t)k * f.ldl];
        }
    }
    __syncthreads();
    // F11bar = tril(S + S'), diagonal S(i, i)
    for (int64_t e = tid; e < (int64_t)c * c; e += nt) {
        const int i = (int)(e % c), j = (int)(e / c);
        if (i < j) continue;
        G[i + (int64_t)j * f.ldl] =
            i == j ? W[i + (int64_t)i * c] : W[i + (int64_t)j * c] + W[j + (int64_t)i * c];
    }
}

__global__ void __launch_bounds__(256)
    k_adj_front(const FrontDesc* __restrict__ fronts, const int* __restrict__ list,
                const double* __restrict__ Ls, double* __restrict__ Fb,
                const double* __restrict__ Fu, const int64_t* __restrict__ zuoff,
                double* __restrict__ Wscr, const int64_t* __restrict__ woff) {
    adj_front(list[blockIdx.x], fronts, Ls, Fb, Fu, zuoff, Wscr, woff);
}

// ---------------------------------------------------------------------------
// large fronts.  The tiles multiply zeros (above the diagonal of an inverse, past
// a front's edge) with the gradients, a NaN where one is infinite or a NaN itself:
// for an Lbar with such entries (odd) every front takes the scalar sums above, in
// the last of its launches.
// ---------------------------------------------------------------------------

struct AdjData {
    const FrontDesc* fronts;
    const double* Ls;
    const double* Dinv;
    const int64_t* dinv_off;
    double* Fb;
    const double* Fu;
    const int64_t* zuoff;
    double* W;      // c x c scratch per front (wide: P, X, S)
    const int64_t* woff;
    double* part;   // 64 x 64 parts of F21bar' L21, by CTA of k_adj_rows
    const int* odd;
    __device__ void scalar_front(int s) const {
        adj_front(s, fronts, Ls, Fb, Fu, zuoff, W, woff);
    }
};
struct AdjList {
    const int* items;
    const int* before;
    int nitems, nctas;
};
// the front of a CTA and its number there
struct AdjJob {
    int s, q;
    FrontDesc f;
    __device__ AdjJob(const AdjData& D, const AdjList& w) {
        const int it = find_item(w.before, w.nitems, blockIdx.x);
        s = w.items[it];
        q = blockIdx.x - w.before[it];
        f = D.fronts[s];
    }
};

// operand (Ubar + Ubar')(a0 + x, k): the stored lower entry (the diagonal
// counted twice by the caller, adj_l21bar)
struct SymU {
    const double* U;
    int ldu, a0, u;
    __device__ __forceinline__ const double* operator()(int k, int x) const {
        const int a = a0 + x;
        if (k >= u || a >= u) return nullptr;
        return a >= k ? U + a + (int64_t)k * ldu : U + k + (int64_t)a * ldu;
    }
};

// acc = sum over b of (Ubar + Ubar')(a0 + row, b) L21(b, col0 + column),
// columns < ncols
template <int MT, int NT>
__device__ void adj_ubar_l21(const FrontDesc& f, const double* L, const double* U, int a0, int col0,
                             int ncols, double* sm, double (&acc)[MT][NT][2][4]) {
    using namespace t64;
    const int u = f.m - f.c;
    const double* L21 = L + f.c + (int64_t)col0 * f.ldl;
    const SymU sym{U, f.ldu, a0, u};
    auto a = op(U, [=](int k, int x) { return sym(k, x); });
    auto b = op(L21, [=](int k, int x) -> const double* {
        return k < u && x < ncols ? L21 + k + (int64_t)x * f.ldl : nullptr;
    });
    zero(acc);
    // columns of Ubar before the end of these rows are stored along the rows
    const int mid = min(a0 + T, u);
    auto a_lo = op(U, [=](int k, int x) -> const double* { return k < mid ? sym(k, x) : nullptr; });
    product<false, true>(sm, 0, mid, a_lo, b, acc);
    if (mid < u) product<true, true>(sm, mid, u, a, b, acc);
}

// L21bar less the sum above at element (a0 + r, col): the diagonal of Ubar
// stands for both triangles, so its entry takes part once more
__device__ __forceinline__ double adj_l21bar(const FrontDesc& f, const double* L, const double* U,
                                             const double* G, int a, int col, double sum) {
    return G[f.c + a + (int64_t)col * f.ldl] - sum -
           U[a + (int64_t)a * f.ldu] * L[f.c + a + (int64_t)col * f.ldl];
}

// MT, NT: 64-column products, or 16-column ones for fronts of c <= 16
template <int MT, int NT>
__device__ void adj_rows(const AdjData& D, const AdjJob& job, int odd, double* adj_sm) {
    using namespace t64;
    const FrontDesc& f = job.f;
    const int c = f.c, u = f.m - c, a0 = T * job.q, rows = min(T, u - a0);
    constexpr int NC = cols<MT>();
    const double* L = D.Ls + f.loff;
    double* G = D.Fb + f.loff;
    const double* U = f.parent >= 0 ? D.Fu + D.zuoff[job.s] : nullptr;
    const double* W = D.Dinv + D.dinv_off[job.s];  // inv(L11), 64 x 64 column-major
    double acc[MT][NT][2][4];
    zero(acc);
    if (U) adj_ubar_l21(f, L, U, a0, 0, c, adj_sm, acc);
    if (odd) return;  // (looked at here: its load is long back)
    // R = L21bar less the sum, as the K-slowest operand [column][row]; W
    // beside it [k][column]
    double* R = adj_sm;
    double* B = adj_sm + T * LD;
    each(acc, [&](int r, int col, double v) {
        double x = 0.0;
        if (r < rows && col < c)
            x = U ? adj_l21bar(f, L, U, G, a0 + r, col, v) : G[c + a0 + r + (int64_t)col * f.ldl];
        R[col * LD + r] = x;
    });
    for (int e = threadIdx.x; e < NC * NC; e += THREADS)
        B[(e % NC) * LD + e / NC] = W[(e % NC) + T * (e / NC)];
    __syncthreads();
    zero(acc);
    for (int k = 0; k < c; k += 16) step16(R + k * LD, B + k * LD, acc);
    __syncthreads();
    // F21bar written and kept as [row][column]; L21's rows [row][column]
    each(acc, [&](int r, int col, double v) {
        const bool in = r < rows && col < c;
        if (in) G[c + a0 + r + (int64_t)col * f.ldl] = v;
        R[r * LD + col] = in ? v : 0.0;
    });
    for (int e = threadIdx.x; e < T * NC; e += THREADS) {
        const int r = e & 63, col = e >> 6;
        B[r * LD + col] = r < rows && col < c ? L[c + a0 + r + (int64_t)col * f.ldl] : 0.0;
    }
    __syncthreads();
    // the part: NC x NC outputs (thin: warp 0's 16 rows are all of them)
    zero(acc);
    if (row0<MT>() < NC)
        for (int k = 0; k < rows; k += 16) step16(R + k * LD, B + k * LD, acc);
    double* p = D.part + (int64_t)blockIdx.x * T * T;
    each(acc, [&](int r, int col, double v) {
        if (r < NC) p[r + T * col] = v;
    });
}

__global__ void __launch_bounds__(t64::THREADS, 3) k_adj_rows(AdjData D, AdjList w) {
    extern __shared__ __align__(16) double adj_sm[];
    const int odd = *D.odd;
    const AdjJob job(D, w);
    if (job.f.c <= 16)
        adj_rows<1, 1>(D, job, odd, adj_sm);
    else
        adj_rows<2, 2>(D, job, odd, adj_sm);
}

// The pivot block of a narrow front: L11bar less the row tiles' parts, then
// P = Phi(L11' L11bar), X = P W, S = W' X, F11bar = tril(S + S').
__global__ void __launch_bounds__(t64::THREADS, 3) k_adj_pivot(AdjData D, AdjList w) {
    using namespace t64;
    extern __shared__ __align__(16) double adj_sm[];
    const int odd = *D.odd, s = w.items[blockIdx.x];
    const FrontDesc f = D.fronts[s];
    const int c = f.c;
    const double* L = D.Ls + f.loff;
    double* G = D.Fb + f.loff;
    const double* W = D.Dinv + D.dinv_off[s];
    double* A = adj_sm;
    double* B = adj_sm + T * LD;
    const int p0 = w.before[blockIdx.x], p1 = w.before[blockIdx.x + 1];
    for (int e = threadIdx.x; e < T * T; e += THREADS) {
        const int k = e & 63, i = e >> 6;
        const bool in = k < c && i < c && k >= i;
        double g = 0.0;
        if (in) {
            g = G[k + (int64_t)i * f.ldl];
            double v = 0.0;
#pragma unroll 4
            for (int p = p0; p < p1; ++p) v += D.part[(int64_t)p * T * T + e];
            g -= v;
        }
        A[k * LD + i] = in ? L[k + (int64_t)i * f.ldl] : 0.0;  // L(k, i)
        B[k * LD + i] = g;                                     // L11bar(k, i)
    }
    if (odd) {
        D.scalar_front(s);
        return;
    }
    __syncthreads();
    // a warp whose rows or columns are all past c has nothing to add
    const bool active = row0<2>() < c && col0<2>() < c;
    Acc acc;
    zero(acc);
    for (int k = 0; active && k < c; k += 16) step16(A + k * LD, B + k * LD, acc);
    __syncthreads();
    // P as [column][row], W as [k][column]
    each(acc, [&](int i, int j, double v) {
        A[j * LD + i] = i < j ? 0.0 : i == j ? 0.5 * v : v;
    });
    for (int e = threadIdx.x; e < T * T; e += THREADS) B[(e & 63) * LD + (e >> 6)] = W[e];
    __syncthreads();
    zero(acc);
    for (int k = 0; active && k < c; k += 16) step16(A + k * LD, B + k * LD, acc);  // X = P W
    __syncthreads();
    each(acc, [&](int i, int j, double v) { A[i * LD + j] = v; });  // [k][column]
    __syncthreads();
    zero(acc);
    for (int k = 0; active && k < c; k += 16) step16(B + k * LD, A + k * LD, acc);  // S = W' X
    __syncthreads();
    each(acc, [&](int i, int j, double v) { A[i * LD + j] = v; });
    __syncthreads();
    for (int e = threadIdx.x; e < T * T; e += THREADS) {
        const int i = e & 63, j = e >> 6;
        if (i >= c || j >= c || i < j) continue;
        G[i + (int64_t)j * f.ldl] = i == j ? A[i * LD + i] : A[i * LD + j] + A[j * LD + i];
    }
}

// wide fronts, step by step -------------------------------------------------

// L21bar -= (Ubar + Ubar') L21: CTA per 64 x 64 tile (row tiles fastest)
__global__ void __launch_bounds__(t64::THREADS, 3) k_adj_w_l21(AdjData D, AdjList w) {
    using namespace t64;
    extern __shared__ __align__(16) double adj_sm[];
    const int odd = *D.odd;
    const AdjJob job(D, w);
    if (odd) return;
    const FrontDesc& f = job.f;
    const int u = f.m - f.c, nrt = (u + T - 1) / T;
    const int a0 = T * (job.q % nrt), c0 = T * (job.q / nrt);
    const int rows = min(T, u - a0), cols = min(T, f.c - c0);
    if (f.parent < 0) return;
    const double* L = D.Ls + f.loff;
    double* G = D.Fb + f.loff;
    const double* U = D.Fu + D.zuoff[job.s];
    Acc acc;
    adj_ubar_l21(f, L, U, a0, c0, cols, adj_sm, acc);
    each(acc, [&](int r, int col, double v) {
        if (r < rows && col < cols)
            G[f.c + a0 + r + (int64_t)(c0 + col) * f.ldl] =
                adj_l21bar(f, L, U, G, a0 + r, c0 + col, v);
    });
}

// 64 rows X of X L11 = M, pivot tiles from kb1 down to 0, in place:
// X_k = (M_k - sum over j > k of X_j L_jk) W_k.  row: the first row's entry in
// column 0, column stride ld.
__device__ void adj_solve_rows(const FrontDesc& f, const double* L, const double* Dk, double* row,
                               int64_t ld, int rows, int kb1, double* sm) {
    using namespace t64;
    const int c = f.c, kend = min(T * (kb1 + 1), c);
    for (int kb = kb1; kb >= 0; --kb) {
        const int k0 = T * kb, nb = min(T, c - k0);
        const double* W = Dk + (int64_t)kb * T * T;
        Acc acc;
        zero(acc);
        auto x = op(row, [=](int k, int r) -> const double* {
            return k < kend && r < rows ? row + r + k * ld : nullptr;
        });
        auto l = op(L, [=](int k, int n) -> const double* {
            return k < kend && n < nb ? L + k + (int64_t)(k0 + n) * f.ldl : nullptr;
        });
        product<false, true>(sm, k0 + T, kend, x, l, acc);
        double* R = sm;
        double* B = sm + T * LD;
        each(acc, [&](int r, int n, double v) {
            R[n * LD + r] = r < rows && n < nb ? row[r + (k0 + n) * ld] - v : 0.0;
        });
        for (int e = threadIdx.x; e < T * T; e += THREADS) B[(e & 63) * LD + (e >> 6)] = W[e];
        __syncthreads();
        zero(acc);
        for (int k = 0; k < nb; k += 16) step16(R + k * LD, B + k * LD, acc);
        each(acc, [&](int r, int n, double v) {
            if (r < rows && n < nb) row[r + (k0 + n) * ld] = v;
        });
        __syncthreads();
    }
}

// F21bar = L21bar L11^-1: CTA per 64 rows
__global__ void __launch_bounds__(t64::THREADS, 3) k_adj_w_f21(AdjData D, AdjList w) {
    extern __shared__ __align__(16) double adj_sm[];
    const int odd = *D.odd;
    const AdjJob job(D, w);
    if (odd) return;
    const FrontDesc& f = job.f;
    const int a0 = t64::T * job.q;
    adj_solve_rows(f, D.Ls + f.loff, D.Dinv + D.dinv_off[job.s], D.Fb + f.loff + f.c + a0, f.ldl,
                   min(t64::T, f.m - f.c - a0), (f.c - 1) / t64::T, adj_sm);
}

// L11bar -= tril(F21bar' L21): CTA per lower tile
__global__ void __launch_bounds__(t64::THREADS, 3) k_adj_w_l11(AdjData D, AdjList w) {
    using namespace t64;
    extern __shared__ __align__(16) double adj_sm[];
    const int odd = *D.odd;
    const AdjJob job(D, w);
    if (odd) return;
    const FrontDesc& f = job.f;
    int bi, bj;
    lower_index(job.q, bi, bj);
    const int c = f.c, u = f.m - c, i0 = T * bi, j0 = T * bj;
    const double* X = D.Fb + f.loff + c + (int64_t)i0 * f.ldl;
    const double* L = D.Ls + f.loff + c + (int64_t)j0 * f.ldl;
    Acc acc;
    zero(acc);
    product<true, true>(adj_sm, 0, u, op(X, [=](int k, int x) -> const double* {
                            return k < u && i0 + x < c ? X + k + (int64_t)x * f.ldl : nullptr;
                        }),
                        op(L, [=](int k, int x) -> const double* {
                            return k < u && j0 + x < c ? L + k + (int64_t)x * f.ldl : nullptr;
                        }),
                        acc);
    double* G = D.Fb + f.loff;
    each(acc, [&](int r, int n, double v) {
        const int i = i0 + r, j = j0 + n;
        if (i < c && i >= j) G[i + (int64_t)j * f.ldl] -= v;
    });
}

// P = Phi(L11' L11bar) into the scratch, zeros above the diagonal of the
// diagonal tiles: CTA per lower tile
__global__ void __launch_bounds__(t64::THREADS, 3) k_adj_w_phi(AdjData D, AdjList w) {
    using namespace t64;
    extern __shared__ __align__(16) double adj_sm[];
    const int odd = *D.odd;
    const AdjJob job(D, w);
    if (odd) return;
    const FrontDesc& f = job.f;
    int bi, bj;
    lower_index(job.q, bi, bj);
    const int c = f.c, i0 = T * bi, j0 = T * bj;
    const double* L = D.Ls + f.loff;
    const double* G = D.Fb + f.loff;
    double* P = D.W + D.woff[job.s];
    Acc acc;
    zero(acc);
    product<true, true>(adj_sm, i0, c, op(L, [=](int k, int x) -> const double* {
                            return k < c && i0 + x <= k ? L + k + (int64_t)(i0 + x) * f.ldl
                                                        : nullptr;
                        }),
                        op(G, [=](int k, int x) -> const double* {
                            return k < c && j0 + x <= k ? G + k + (int64_t)(j0 + x) * f.ldl
                                                        : nullptr;
                        }),
                        acc);
    each(acc, [&](int r, int n, double v) {
        const int i = i0 + r, j = j0 + n;
        if (i < c && j < c) P[i + (int64_t)j * c] = i < j ? 0.0 : i == j ? 0.5 * v : v;
    });
}

// X = P L11^-1 in the scratch's lower tiles: CTA per 64 rows
__global__ void __launch_bounds__(t64::THREADS, 3) k_adj_w_x(AdjData D, AdjList w) {
    extern __shared__ __align__(16) double adj_sm[];
    const int odd = *D.odd;
    const AdjJob job(D, w);
    if (odd) return;
    const FrontDesc& f = job.f;
    const int i0 = t64::T * job.q;
    adj_solve_rows(f, D.Ls + f.loff, D.Dinv + D.dinv_off[job.s], D.W + D.woff[job.s] + i0, f.c,
                   min(t64::T, f.c - i0), job.q, adj_sm);
}

// S = L11^-T X in the scratch, all of it: CTA per 64 columns, pivot tiles from
// the last up: S_k = W_k' (X_k - sum over r > k of L_rk' S_r), X_k = 0 above
// the column tile
__global__ void __launch_bounds__(t64::THREADS, 3) k_adj_w_s(AdjData D, AdjList w) {
    using namespace t64;
    extern __shared__ __align__(16) double adj_sm[];
    const int odd = *D.odd;
    const AdjJob job(D, w);
    if (odd) return;
    const FrontDesc& f = job.f;
    const int c = f.c, j0 = T * job.q, cols = min(T, c - j0);
    const double* L = D.Ls + f.loff;
    double* S = D.W + D.woff[job.s] + (int64_t)j0 * c;
    for (int kb = (c - 1) / T; kb >= 0; --kb) {
        const int k0 = T * kb, nb = min(T, c - k0);
        const double* W = D.Dinv + D.dinv_off[job.s] + (int64_t)kb * T * T;
        Acc acc;
        zero(acc);
        product<true, true>(adj_sm, k0 + T, c, op(L, [=](int k, int x) -> const double* {
                                return k < c && x < nb ? L + k + (int64_t)(k0 + x) * f.ldl
                                                       : nullptr;
                            }),
                            op(S, [=](int k, int x) -> const double* {
                                return k < c && x < cols ? S + k + (int64_t)x * c : nullptr;
                            }),
                            acc);
        double* R = adj_sm;           // [k][column]
        double* B = adj_sm + T * LD;  // W(k, i) as [k][i]
        each(acc, [&](int r, int n, double v) {
            double x = 0.0;
            if (r < nb && n < cols) x = (kb >= job.q ? S[k0 + r + (int64_t)n * c] : 0.0) - v;
            R[r * LD + n] = x;
        });
        for (int e = threadIdx.x; e < T * T; e += THREADS) B[(e & 63) * LD + (e >> 6)] = W[e];
        __syncthreads();
        zero(acc);
        for (int k = 0; k < nb; k += 16) step16(B + k * LD, R + k * LD, acc);
        each(acc, [&](int r, int n, double v) {
            if (r < nb && n < cols) S[k0 + r + (int64_t)n * c] = v;
        });
        __syncthreads();
    }
}

// F11bar = tril(S + S'), diagonal S(i, i): CTA per lower tile
__global__ void __launch_bounds__(t64::THREADS) k_adj_w_f11(AdjData D, AdjList w) {
    using namespace t64;
    __shared__ double tr[T][T + 1];
    const int odd = *D.odd;
    const AdjJob job(D, w);
    if (odd) {
        if (job.q == 0) D.scalar_front(job.s);
        return;
    }
    const FrontDesc& f = job.f;
    int bi, bj;
    lower_index(job.q, bi, bj);
    const int c = f.c, i0 = T * bi, j0 = T * bj;
    const double* S = D.W + D.woff[job.s];
    double* G = D.Fb + f.loff;
    for (int e = threadIdx.x; e < T * T; e += THREADS) {
        const int j = e & 63, i = e >> 6;  // S(j0 + j, i0 + i), read down its column
        tr[i][j] = i0 + i < c && j0 + j < c ? S[j0 + j + (int64_t)(i0 + i) * c] : 0.0;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < T * T; e += THREADS) {
        const int i = i0 + (e & 63), j = j0 + (e >> 6);
        if (i >= c || j >= c || i < j) continue;
        const double v = S[i + (int64_t)j * c];
        G[i + (int64_t)j * f.ldl] = i == j ? v : v + tr[i - i0][j - j0];
    }
}

// Abar of every lower-triangle entry e (caller order; zeroed by the caller):
// Fbar at the front position the assembly gave it
__global__ void k_adj_abar(int nnz, const FrontDesc* __restrict__ fronts,
                           const int* __restrict__ a_front, const int* __restrict__ a_src,
                           const int* __restrict__ a_pos, const double* __restrict__ Fb,
                           double* __restrict__ Abar) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += gridDim.x * blockDim.x) {
        const int src = a_src[e];
        if (src < 0) continue;  // a duplicate the assembly drops: gradient 0
        const FrontDesc f = fronts[a_front[e]];
        const int pos = a_pos[e], r = pos & 0xffff, jj = pos >> 16;
        Abar[src] = Fb[f.loff + r + (int64_t)jj * f.ldl];
    }
}

// CTAs of the largest k_adj_rows launch: the 64 x 64 parts it keeps, and the odd
// flag's place behind them
int64_t adjoint_parts(const DevPlan& D) {
    int64_t p = 1;
    for (const AdjLevel& l : D.adj.h_large) p = std::max<int64_t>(p, l.rows.nctas);
    return p * t64::T * t64::T + 1;
}

void launch_adjoint(const DevPlan& D, int nnz, const double* Ls, const double* Dinv,
                    const double* Lbar, double* Fb, double* Fu, double* Wscr, double* part,
                    double* Abar, cudaStream_t st) {
    const AdjSchedule& S = D.adj;
    constexpr size_t SM = t64::SMEM_BYTES;
    int* odd = reinterpret_cast<int*>(part + adjoint_parts(D) - 1);
    cudaMemsetAsync(odd, 0, sizeof(int), st);
    const int sms = D.num_sms > 0 ? D.num_sms : 148;
    k_adj_check<<<(int)std::min<int64_t>((S.lnz + 1023) / 1024, 8 * sms), 256, 0, st>>>(S.lnz, Lbar,
                                                                                       odd);
    const AdjData data{D.fronts, Ls, Dinv, D.dinv_off, Fb, Fu, D.zuoff, Wscr, S.woff, part, odd};
    auto list = [&](const WorkList& w) {
        return AdjList{S.items + w.off, S.before + w.off, w.nitems, w.nctas};
    };
    const int nsmall = D.h_small_ptr[D.nlevels * kSmallBuckets], nlarge = D.h_large_ptr[D.nlevels];
    if (nsmall > 0)
        k_adj_scatter<<<nsmall, 64, 0, st>>>(D.fronts, D.small_list, S.Lp, Lbar, Fb);
    if (nlarge > 0)
        k_adj_scatter<<<dim3(nlarge, 8), 256, 0, st>>>(D.fronts, D.large_list, S.Lp, Lbar, Fb);
    for (int l = D.nlevels - 1; l >= 0; --l) {
        const WorkList& g = S.h_gather[l];
        if (g.nctas > 0)
            k_adj_gather<<<g.nctas, 256, 0, st>>>(D.fronts, S.items + g.off, S.before + g.off,
                                                  g.nitems, D.relmap, Fb, Fu, D.zuoff);
        // the level's small fronts beside its large ones
        const int b = D.h_small_ptr[l * kSmallBuckets], e = D.h_small_ptr[(l + 1) * kSmallBuckets];
        const AdjLevel& A = S.h_large[l];
        const bool fork = e > b && (A.rows.nitems > 0 || A.wide_rows.nitems > 0) && D.piece_st[0];
        const cudaStream_t ss = fork ? D.piece_st[0] : st;
        if (fork) {
            cudaEventRecord(D.fork_ev, st);
            cudaStreamWaitEvent(ss, D.fork_ev, 0);
        }
        if (e > b)
            k_adj_front<<<e - b, 256, 0, ss>>>(D.fronts, D.small_list + b, Ls, Fb, Fu, D.zuoff,
                                               Wscr, S.woff);
        if (fork) cudaEventRecord(D.piece_join[0], ss);
        if (A.rows.nctas > 0) k_adj_rows<<<A.rows.nctas, t64::THREADS, SM, st>>>(data, list(A.rows));
        if (A.rows.nitems > 0)
            k_adj_pivot<<<A.rows.nitems, t64::THREADS, SM, st>>>(data, list(A.rows));
        if (A.wide_rows.nitems > 0) {
            if (A.wide_l21.nctas > 0) {
                k_adj_w_l21<<<A.wide_l21.nctas, t64::THREADS, SM, st>>>(data, list(A.wide_l21));
                k_adj_w_f21<<<A.wide_rows.nctas, t64::THREADS, SM, st>>>(data, list(A.wide_rows));
                k_adj_w_l11<<<A.wide_low.nctas, t64::THREADS, SM, st>>>(data, list(A.wide_low));
            }
            k_adj_w_phi<<<A.wide_low.nctas, t64::THREADS, SM, st>>>(data, list(A.wide_low));
            k_adj_w_x<<<A.wide_piv.nctas, t64::THREADS, SM, st>>>(data, list(A.wide_piv));
            k_adj_w_s<<<A.wide_piv.nctas, t64::THREADS, SM, st>>>(data, list(A.wide_piv));
            k_adj_w_f11<<<A.wide_low.nctas, t64::THREADS, 0, st>>>(data, list(A.wide_low));
        }
        if (fork) cudaStreamWaitEvent(st, D.piece_join[0], 0);
    }
    cudaMemsetAsync(Abar, 0, (size_t)nnz * sizeof(double), st);
    const int blocks = std::max(1, std::min((nnz + 255) / 256, 148 * 8));
    k_adj_abar<<<blocks, 256, 0, st>>>(nnz, D.fronts, D.a_front, D.a_src, D.a_pos, Fb, Abar);
}

void init_adjoint() {
    const int sm = (int)t64::SMEM_BYTES;
    for (auto* k : {k_adj_rows, k_adj_pivot, k_adj_w_l21, k_adj_w_f21, k_adj_w_l11, k_adj_w_phi,
                    k_adj_w_x, k_adj_w_s})
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
}

}  // namespace mdgpu
