// 64 x 64 tile operations shared by the large-front factor kernels: the
// diagonal-tile Cholesky with its inverse, and the register-tiled products
// C -= A B' over 256 threads (a 4 x 4 block of outputs each).
#pragma once

#include <cuda_runtime.h>

#include "device_common.cuh"

namespace mdgpu {

__device__ __forceinline__ float recip_sqrt(float x) { return rsqrtf(x); }
__device__ __forceinline__ double recip_sqrt(double x) { return rsqrt(x); }

// Leading dimension of the diagonal-tile factorization's S and W: a 4x4
// block's columns are 16-byte vectors (4 floats or 2 x 2 doubles).
constexpr int kPotrfLD = 64 + 4;

// a 4x4 block at (r0, c0) of a kPotrfLD column-major array, in and out
template <typename T>
__device__ __forceinline__ void blk_ld(const T* M, int r0, int c0, T (&b)[4][4]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const T* p = M + r0 + (c0 + c) * kPotrfLD;
        if constexpr (sizeof(T) == 4) {
            const float4 v = *reinterpret_cast<const float4*>(p);
            b[0][c] = v.x, b[1][c] = v.y, b[2][c] = v.z, b[3][c] = v.w;
        } else {
            const double2 v0 = *reinterpret_cast<const double2*>(p);
            const double2 v1 = *reinterpret_cast<const double2*>(p + 2);
            b[0][c] = v0.x, b[1][c] = v0.y, b[2][c] = v1.x, b[3][c] = v1.y;
        }
    }
}
template <typename T>
__device__ __forceinline__ void blk_st(T* M, int r0, int c0, const T (&b)[4][4]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        T* p = M + r0 + (c0 + c) * kPotrfLD;
        if constexpr (sizeof(T) == 4) {
            *reinterpret_cast<float4*>(p) = make_float4(b[0][c], b[1][c], b[2][c], b[3][c]);
        } else {
            *reinterpret_cast<double2*>(p) = make_double2(b[0][c], b[1][c]);
            *reinterpret_cast<double2*>(p + 2) = make_double2(b[2][c], b[3][c]);
        }
    }
}

// Factor a 4x4 diagonal block in registers: a -> L (lower, zeros above), y =
// inv(L).  One reciprocal square root per pivot (d = piv / sqrt(piv)); the
// first non-positive (or NaN) pivot of a row < n is recorded at global column
// col0 + row0 + i, after the four pivots (no branch on their chain).
template <typename T>
__device__ __forceinline__ void diag4(T (&a)[4][4], T (&y)[4][4], int row0, int n, int col0,
                                      int* status) {
    int bad = 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const T piv = a[i][i];
        if (!(piv > T(0))) bad = min(bad, i);
        const T rd = recip_sqrt(piv);
        a[i][i] = piv * rd;
        y[i][i] = rd;
#pragma unroll
        for (int r = i + 1; r < 4; ++r) a[r][i] *= rd;
#pragma unroll
        for (int r = i + 1; r < 4; ++r)
#pragma unroll
            for (int c = i + 1; c <= r; ++c) a[r][c] -= a[r][i] * a[c][i];
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int r = c + 1; r < 4; ++r) {
            T v = T(0);
#pragma unroll
            for (int m = c; m < r; ++m) v -= a[r][m] * y[m][c];
            y[r][c] = v * y[r][r];
        }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = r + 1; c < 4; ++c) a[r][c] = y[r][c] = T(0);
    if (row0 + bad < n && bad < 4) flag_pivot(status, col0 + row0 + bad);
}

// barrier of the first `threads` threads of the CTA (whole warps)
__device__ __forceinline__ void part_sync(int id, int threads) {
    asm volatile("barrier.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

template <typename T>
__device__ __forceinline__ void vec4_ld(const T* p, T& a, T& b, T& c, T& d) {
    if constexpr (sizeof(T) == 4) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        a = v.x, b = v.y, c = v.z, d = v.w;
    } else {
        const double2 v = *reinterpret_cast<const double2*>(p);
        const double2 w = *reinterpret_cast<const double2*>(p + 2);
        a = v.x, b = v.y, c = w.x, d = w.y;
    }
}
template <typename T>
__device__ __forceinline__ void vec4_st(T* p, T a, T b, T c, T d) {
    if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
    } else {
        *reinterpret_cast<double2*>(p) = make_double2(a, b);
        *reinterpret_cast<double2*>(p + 2) = make_double2(c, d);
    }
}
// o = a y' for a lower triangular y
template <typename T>
__device__ __forceinline__ void mul_yt(const T (&a)[4][4], const T (&y)[4][4], T (&o)[4][4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            T v = T(0);
#pragma unroll
            for (int m = 0; m <= c; ++m) v += a[r][m] * y[c][m];
            o[r][c] = v;
        }
}

// Cholesky of the TB x TB tile held in S (lower part; a partial tile of n <
// TB rows padded with the identity) and its inverse.  On exit S holds L and W
// inv(L), both in the lower 4 x 4 blocks of the first ceil(n / 4) block rows
// (nothing else of W is written, and the rest of S is left alone: the steps
// past the tile's own rows are not taken).  S, W: TB x kPotrfLD, column-major.
// The tile is a 16 x 16 grid of 4 x 4 blocks.  Threads 0..119 own the
// strictly lower blocks (column by column: block (tr, tc) and its block of X
// = inv(L)), threads 128..143 the diagonal blocks; thread 160 alone factors
// the diagonal blocks, one step ahead of the others, so that the chain of
// square roots runs beside their work.  Step kb (the diagonal block kb is
// factored, its L in S and its inverse Y in W and in thread 160's registers):
//   thread 160   forms P = A(kb + 1, kb) Y', takes P P' off diagonal block
//                kb + 1 and factors it; both blocks come through `hand`
//                (two slots, by step parity) from their owners, updated
//                through step kb - 1;
//   the owners   (1) block column kb: P = A Y' to S; block row kb of X: Y x
//                to W; then, after a barrier of their own, (2) the blocks
//                right of kb take the rank-4 update with the panel (the two
//                that thread 160 needs next go to `hand`), the X blocks below
//                x -= L(tr, kb) X(kb, tc).
// Latency-bound (one warp per scheduler at a third of the issue rate): 17 k
// cycles for a whole FP32 tile, 4.4 k for 16 rows, 1.6 k for one.
// Starts and ends with a CTA barrier; uses named barriers 1 and 2.
template <typename T, int TB>
__device__ void potrf_tile_core(T* S, T* W, int n, int col0, int* status) {
    static_assert(TB == 64 && TB + 4 == kPotrfLD, "16 x 16 grid of 4 x 4 blocks over 256 threads");
    constexpr int B = 4, NB = TB / B, NSTRICT = NB * (NB - 1) / 2, DIAG0 = 128, CHAIN = 160,
                  OWNERS = 160, ALL = 192;
    // slot, {A(kb + 1, kb), A(kb + 1, kb + 1)}, column-major
    __shared__ __align__(16) T hand[2][2][B * B];
    const int tid = threadIdx.x, nb = (n + B - 1) / B;
    const bool strict = tid < NSTRICT;
    const bool diag = tid >= DIAG0 && tid < DIAG0 + NB;
    int tr = 0, tc = 0;
    if (strict) {  // column-major order of the strictly lower blocks
        int p = tid;
        while (p >= NB - 1 - tc) p -= NB - 1 - tc, ++tc;
        tr = tc + 1 + p;
    } else if (diag) {
        tr = tc = tid - DIAG0;
    }
    const bool mine = (strict || diag) && tr < nb;
    auto give = [&](int slot, const T (&v)[B][B]) {
#pragma unroll
        for (int c = 0; c < B; ++c)
            vec4_st(hand[slot][diag ? 1 : 0] + c * B, v[0][c], v[1][c], v[2][c], v[3][c]);
    };
    auto take = [&](int slot, int which, T (&v)[B][B]) {
#pragma unroll
        for (int c = 0; c < B; ++c)
            vec4_ld(hand[slot][which] + c * B, v[0][c], v[1][c], v[2][c], v[3][c]);
    };
    __syncthreads();
    T a[B][B], x[B][B], y[B][B];
#pragma unroll
    for (int r = 0; r < B; ++r)
#pragma unroll
        for (int c = 0; c < B; ++c) a[r][c] = x[r][c] = T(0);
    if (mine || tid == CHAIN) blk_ld(S, B * tr, B * tc, a);
    if (mine && tr == 1) give(0, a);
    __syncthreads();
    if (tid < ALL) {
        if (tid == CHAIN) {
            diag4(a, y, 0, n, col0, status);
            blk_st(S, 0, 0, a);
            blk_st(W, 0, 0, y);
        }
        part_sync(2, ALL);
#pragma unroll 1
        for (int kb = 0; kb < nb; ++kb) {
            if (tid >= OWNERS) {
                if (tid == CHAIN && kb + 1 < nb) {
                    T p[B][B], q[B][B];
                    take(kb & 1, 0, p);
                    take(kb & 1, 1, a);
                    mul_yt(p, y, q);
#pragma unroll
                    for (int r = 0; r < B; ++r)
#pragma unroll
                        for (int c = 0; c <= r; ++c)
#pragma unroll
                            for (int m = 0; m < B; ++m) a[r][c] -= q[r][m] * q[c][m];
                    diag4(a, y, B * (kb + 1), n, col0, status);
                    blk_st(W, B * (kb + 1), B * (kb + 1), y);
                    blk_st(S, B * (kb + 1), B * (kb + 1), a);
                }
            } else {
                if (mine && strict && (tc == kb || tr == kb)) {  // (1)
                    T o[B][B];
                    blk_ld(W, B * kb, B * kb, y);
                    if (tc == kb) {  // panel block: A Y'
                        mul_yt(a, y, o);
                        blk_st(S, B * tr, B * kb, o);
                    } else {  // inverse block row kb: Y x
#pragma unroll
                        for (int r = 0; r < B; ++r)
#pragma unroll
                            for (int c = 0; c < B; ++c) {
                                T v = T(0);
#pragma unroll
                                for (int m = 0; m <= r; ++m) v += y[r][m] * x[m][c];
                                o[r][c] = v;
                            }
                        blk_st(W, B * kb, B * tc, o);
                    }
                }
                part_sync(1, OWNERS);
                if (mine && tr > kb) {  // (2)
                    T p[B][B], q[B][B];
                    blk_ld(S, B * tr, B * kb, p);
                    if (tc > kb) {  // trailing update with the panel
                        blk_ld(S, B * tc, B * kb, q);
#pragma unroll
                        for (int r = 0; r < B; ++r)
#pragma unroll
                            for (int c = 0; c < B; ++c)
#pragma unroll
                                for (int m = 0; m < B; ++m) a[r][c] -= p[r][m] * q[c][m];
                        if (tr == kb + 2) give((kb + 1) & 1, a);
                    } else {  // inverse rows below: x -= L(tr, kb) X(kb, tc)
                        blk_ld(W, B * kb, B * tc, q);
#pragma unroll
                        for (int r = 0; r < B; ++r)
#pragma unroll
                            for (int c = 0; c < B; ++c)
#pragma unroll
                                for (int m = 0; m < B; ++m) x[r][c] -= p[r][m] * q[m][c];
                    }
                }
            }
            part_sync(2, ALL);
        }
    }
    __syncthreads();
}

// acc = sum over q < K of As[q][r0 + a] * Bs[q][c0 + b] (As, Bs: K x TB,
// row q at q * TB), r0 = 4 (tid mod 16), c0 = 4 (tid / 16).
template <typename T, int TB>
__device__ void tile_gemm_nt_acc(const T* As, const T* Bs, int K, T (&acc)[4][4]) {
    const int tid = threadIdx.x;
    const int r0 = (tid & 15) * 4, c0 = (tid >> 4) * 4;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = T(0);
    for (int q = 0; q < K; ++q) {
        T av[4], bv[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) av[a] = As[q * TB + r0 + a];
#pragma unroll
        for (int b = 0; b < 4; ++b) bv[b] = Bs[q * TB + c0 + b];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a][b] += av[a] * bv[b];
    }
}

// a thread's four rows (or columns) of step q of a K x TB block
template <typename T>
__device__ __forceinline__ void frag4(const T* p, T (&v)[4]) {
    vec4_ld(p, v[0], v[1], v[2], v[3]);
}

// acc += the full-K (TB) product of two TB x TB blocks, as tile_gemm_nt_acc;
// both blocks 16-byte aligned, so each thread reads its four rows and four
// columns of a K step with vector loads.
template <typename T, int TB>
__device__ __forceinline__ void tile_gemm_nt_add(const T* __restrict__ As,
                                                 const T* __restrict__ Bs, T (&acc)[4][4]) {
    const int tid = threadIdx.x;
    const int r0 = (tid & 15) * 4, c0 = (tid >> 4) * 4;
    constexpr int U = 2;  // steps loaded ahead of their products
    T av[2][U][4], bv[2][U][4];
#pragma unroll
    for (int q = 0; q < U; ++q) {
        frag4(As + q * TB + r0, av[0][q]);
        frag4(Bs + q * TB + c0, bv[0][q]);
    }
#pragma unroll 4
    for (int q0 = 0; q0 < TB; q0 += U) {
        const int s = (q0 / U) & 1;
        if (q0 + U < TB) {
#pragma unroll
            for (int q = 0; q < U; ++q) {
                frag4(As + (q0 + U + q) * TB + r0, av[s ^ 1][q]);
                frag4(Bs + (q0 + U + q) * TB + c0, bv[s ^ 1][q]);
            }
        }
#pragma unroll
        for (int q = 0; q < U; ++q)
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] += av[s][q][a] * bv[s][q][b];
    }
}

// The column group of a thread in tile_gemm_tri: warp w's eight columns, the
// warps of one scheduler (w and w + 4) taking a short and a long one.
__device__ __forceinline__ int tri_c0(int tid) {
    const int w = tid >> 5;
    return 8 * (w < 4 ? w : 11 - w) + 4 * ((tid >> 4) & 1);
}

// As tile_gemm_nt_add for Bs[q][c] zero where q > c (the transposed inverse
// of a lower triangular tile) or q >= K, at rows 4 (tid mod 16) and columns
// tri_c0(tid): a warp stops at its own last column.  (FP32; FP64 products run on
// the matrix instructions.)
template <int TB>
__device__ __forceinline__ void tile_gemm_tri(const float* __restrict__ As,
                                              const float* __restrict__ Bs, int K,
                                              float (&acc)[4][4]) {
    const int tid = threadIdx.x;
    const int r0 = (tid & 15) * 4, c0 = tri_c0(tid);
    const int qn = min((c0 & ~7) + 8, (K + 3) & ~3);
#pragma unroll 4
    for (int q = 0; q < qn; ++q) {
        const float4 a4 = *reinterpret_cast<const float4*>(As + q * TB + r0);
        const float4 b4 = *reinterpret_cast<const float4*>(Bs + q * TB + c0);
        const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a][b] += av[a] * bv[b];
    }
}

}  // namespace mdgpu
