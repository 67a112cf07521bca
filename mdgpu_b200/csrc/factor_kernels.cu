// Numeric factorization kernels (scalar T = double or float).
//
// Small fronts (m <= 160): a CTA, a warp or a part of a warp per front does
// everything in shared memory and registers: zero the front, scatter A's values,
// extend-add every child's update matrix (children one after another, so the
// sum is deterministic), factor the c pivot columns, write the L panel and the
// Schur complement U = F22 - L21 L21'.
//
// Large fronts: a tiled right-looking partial Cholesky over the [L | U] split
// storage, batched over all large fronts of one tree level:
//   k_big_assemble_warp  CTA per (front, 16-column block), a warp per column: A's
//                    values and the children's update columns that land in it
//                    (k_big_assemble: the same for the 64-wide schedule below)
//   k_panel, k_schur_*   (files of their own) the pivot columns in panels of 256,
//                    each followed by one update of the trailing part
// FP32 factors with no TMA descriptors step by single tiles instead:
//   k_tile_potrf     CTA per front: Cholesky of the first diagonal tile, and its
//                    inverse (kept: it turns every TRSM and every solve step
//                    with this tile into a small matrix product)
//   k_tile_trsm      CTA per (front, row tile below the panel): X = A inv(L)'
//   k_tile_update    CTA per (front, lower tile right of the panel):
//                    C -= A B'; the CTA holding the next diagonal tile also
//                    factors it, so the next step's TRSM can start at once.
#include <cstdio>

#include "device_common.cuh"
#include "kernels.hpp"
#include "tile_ops.cuh"

namespace mdgpu {

// ---------------------------------------------------------------------------
// small fronts
// ---------------------------------------------------------------------------

// Most small fronts have one to a few pivot columns, so their time is the
// chain of dependent memory trips and barriers of the assembly, not
// arithmetic: descriptions of up to 32 children are loaded by the lanes at
// once, a warp takes eight columns of a child's update matrix at a time, lane =
// row, with the next eight on their way, across children too, and no index is
// divided.  (With a division per element, a barrier or two per child and per
// pivot column: fronts of 33..160 rows 11.5 ms, now 4.2, and up to 32 rows 1.1,
// now 0.74, over 130 + 26 launches of a batch of 2D and 3D grids, FP32; a root
// of 149 columns FP64 478 us, now 85.)  What is left of a level of a few tiny
// fronts, 4 to 8 us, is mostly its cold instructions: about ten cycles each.

// (correctly rounded both: a reciprocal square root with a Newton step for each
// took 1 to 2 % less of the kernels' time, and moved L by roundings)
template <typename T>
__device__ __forceinline__ void pivot_root(T x, T& root, T& inv) {
    root = sqrt(x);
    inv = T(1) / root;
}

// 8 neighbouring elements on 16 bytes
__device__ __forceinline__ void vec8_ld(const float* p, float (&v)[8]) {
    const float4 a = reinterpret_cast<const float4*>(p)[0];
    const float4 b = reinterpret_cast<const float4*>(p)[1];
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
__device__ __forceinline__ void vec8_ld(const double* p, double (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double2 a = reinterpret_cast<const double2*>(p)[i];
        v[2 * i] = a.x, v[2 * i + 1] = a.y;
    }
}

// leading dimension of a front of up to MB rows in shared memory (columns on
// 16 bytes)
template <typename T>
__host__ __device__ constexpr int small_ld(int MB) {
    return MB + 16 / (int)sizeof(T);
}

// One front of up to MB rows by `nw` warps (ceil(MB / 32) or fewer, up to the
// block's), F: MB columns of LD = small_ld(MB) elements; sync: a barrier over
// the nw warps.
template <typename T, typename Sync>
__device__ __forceinline__ void small_front(const FrontDesc& f, T* F, int LD, int warp, int nw,
                                            Sync&& sync, const FrontDesc* __restrict__ fronts,
                                            const int* __restrict__ child,
                                            const int* __restrict__ relmap,
                                            const int* __restrict__ a_src,
                                            const int* __restrict__ a_pos,
                                            const double* __restrict__ Ax, T* __restrict__ Ls,
                                            T* __restrict__ Us, int* __restrict__ status) {
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int CG = 8;  // columns at a time: most fronts' pivot columns fit one panel
    const int m = f.m, c = f.c, lane = threadIdx.x & 31;
    const int tid = 32 * warp + lane, nt = 32 * nw;
    // the chains of loads before the first barrier side by side: an A entry's
    // place and value, and child, description, update matrix
    int src = -1, pos = 0;
    if (f.a_beg + tid < f.a_end) {
        src = a_src[f.a_beg + tid];
        pos = a_pos[f.a_beg + tid];
    }
    int g_id = -1;
    if (f.child_beg + lane < f.child_end) g_id = child[f.child_beg + lane];
    for (int idx = tid; idx < m * LD * (int)sizeof(T) / 16; idx += nt)
        reinterpret_cast<int4*>(F)[idx] = make_int4(0, 0, 0, 0);

    // the children of a batch of up to 32, one per lane
    int64_t g_u = 0;
    int g_uc = 0, g_ldu = 0, g_rel = 0;
    // the trip of this warp: CG columns from j0 on of child h of the batch, rows
    // i0 + lane; h == nb at the end
    int hb = f.child_beg, nb = 0, h = 0, j0 = 0, i0 = 0, uc = 0;
    auto settle = [&]() {  // skips children with no trip left
        while (j0 >= uc) {
            if (++h >= nb) return;
            uc = __shfl_sync(ALL, g_uc, h);
            j0 = CG * warp;
            i0 = j0 & ~31;
        }
    };
    auto describe = [&]() {
        nb = min(32, f.child_end - hb);
        g_uc = 0;
        if (g_id >= 0) {
            const FrontDesc& g = fronts[g_id];
            g_uc = g.m - g.c;
            g_ldu = g.ldu;
            g_rel = g.rows_off + g.c;
            g_u = g.uoff;
        }
    };
    auto begin = [&]() {
        h = -1, j0 = uc = 0;
        settle();
    };
    T v[CG];
    int ri = 0, rj = 0;  // the trip's row of this lane, column of lane & 7
    auto fetch = [&]() {
        if (h >= nb) return;
        const T* U = Us + __shfl_sync(ALL, g_u, h);
        const int ldu = __shfl_sync(ALL, g_ldu, h);
        const int* rm = relmap + __shfl_sync(ALL, g_rel, h);
        const int i = i0 + lane;
#pragma unroll
        for (int e = 0; e < CG; ++e) {
            v[e] = T(0);
            if (i < uc && i >= j0 + e) v[e] = U[i + (int64_t)(j0 + e) * ldu];
        }
        ri = i < uc ? rm[i] : 0;
        rj = j0 + (lane & 7) < uc ? rm[j0 + (lane & 7)] : 0;
    };
    describe();
    const T av = src >= 0 ? (T)Ax[src] : T(0);
    begin();
    fetch();
    sync();
    if (src >= 0) F[(pos & 0xffff) + (pos >> 16) * LD] = av;
    for (int e = f.a_beg + nt + tid; e < f.a_end; e += nt) {
        src = a_src[e];
        if (src >= 0) {
            pos = a_pos[e];
            F[(pos & 0xffff) + (pos >> 16) * LD] = (T)Ax[src];
        }
    }
    // children in order, a barrier after each
    for (;;) {
        for (int done = -1; done < nb;) {
            // to the child of the trip at hand
            for (; done < h; ++done) sync();
            if (h >= nb) break;
            T w[CG];
#pragma unroll
            for (int e = 0; e < CG; ++e) w[e] = v[e];
            const int wi = ri, wj = rj, cnt = uc, i = i0 + lane, jb = j0;
            i0 += 32;
            if (i0 >= uc) {
                j0 += CG * nw;
                i0 = j0 & ~31;
                settle();
            }
            fetch();
            T* at[CG];  // distinct columns: all reads before the writes
#pragma unroll
            for (int e = 0; e < CG; ++e) {
                at[e] = F + wi + __shfl_sync(ALL, wj, e) * LD;
                if (i < cnt && i >= jb + e) w[e] += *at[e];
            }
#pragma unroll
            for (int e = 0; e < CG; ++e)
                if (i < cnt && i >= jb + e) *at[e] = w[e];
        }
        hb += 32;
        if (hb >= f.child_end) break;
        g_id = hb + lane < f.child_end ? child[hb + lane] : -1;
        describe();
        begin();
        fetch();
    }

    // pivot columns in panels of eight, lane = row, every warp factoring the
    // diagonal block along with its rows (its multipliers by shuffles), then the
    // trailing update; the last panel's goes straight to the update store
    for (int p = 0; p < c; p += CG) {
        const int n = min(CG, c - p), pe = p + n;
        T a[CG];
        // (the first block last: its diagonal rows wait for the barrier)
        const int nrb = (m - p + 31) / 32;
        for (int rb = warp + (nrb - 1 - warp) / nw * nw; warp < nrb && rb >= 0; rb -= nw) {
            const int r = p + 32 * rb + lane;
            T d[CG];
#pragma unroll
            for (int j = 0; j < CG; ++j) {
                d[j] = a[j] = T(0);
                if (j < n) {
                    d[j] = F[p + (lane & 7) + (p + j) * LD];
                    if (r < m) a[j] = F[r + (p + j) * LD];
                }
            }
#pragma unroll
            for (int k = 0; k < CG; ++k) {
                if (k >= n) break;
                const T piv = __shfl_sync(ALL, d[k], k);
                T root, inv;
                pivot_root(piv, root, inv);
                if (rb == 0 && lane == k && !(piv > T(0))) flag_pivot(status, f.first_col + p + k);
                const T ld = d[k] * inv, lr = a[k] * inv;
                a[k] = r == p + k ? root : lr;
#pragma unroll
                for (int j = k + 1; j < CG; ++j) {
                    const T t = __shfl_sync(ALL, ld, j);
                    d[j] -= ld * t;
                    a[j] -= lr * t;
                }
            }
            if (r >= pe && r < m)
#pragma unroll
                for (int j = 0; j < CG; ++j)
                    if (j < n) F[r + (p + j) * LD] = a[j];
        }
        sync();
        if (warp == 0 && lane < n)
#pragma unroll
            for (int j = 0; j < CG; ++j)
                if (j <= lane) F[p + lane + (p + j) * LD] = a[j];
        const bool last = pe == c;
        if (last && f.uoff < 0) break;
        for (int jg = (pe & ~(CG - 1)) + CG * warp; jg < m; jg += CG * nw) {
            // rows from the first one on or below the group's diagonal
            for (int r0 = max(jg, pe); r0 < m; r0 += 32) {
                const int r = r0 + lane;
                T acc[CG];
#pragma unroll
                for (int e = 0; e < CG; ++e) acc[e] = r < m ? F[r + (jg + e) * LD] : T(0);
#pragma unroll 4
                for (int k = p; k < pe; ++k) {
                    T b[CG];
                    vec8_ld(F + jg + k * LD, b);
                    const T x = r < m ? F[r + k * LD] : T(0);
#pragma unroll
                    for (int e = 0; e < CG; ++e) acc[e] -= x * b[e];
                }
#pragma unroll
                for (int e = 0; e < CG; ++e) {
                    const int j = jg + e;
                    if (r >= m || r < j || j < pe) continue;
                    if (last)
                        Us[f.uoff + (r - c) + (int64_t)(j - c) * f.ldu] = acc[e];
                    else
                        F[r + j * LD] = acc[e];
                }
            }
        }
        if (!last) sync();
    }
    sync();
    for (int j = warp; j < c; j += nw) {
        T* Lj = Ls + f.loff + (int64_t)j * f.ldl;
        for (int r = lane; r < m; r += 32) Lj[r] = r >= j ? F[r + j * LD] : T(0);
    }
}

// Fronts of 33..160 rows: a CTA each.
template <typename T>
__global__ void __launch_bounds__(512)
    k_small_front(const FrontDesc* __restrict__ fronts, const int* __restrict__ list,
                  const int* __restrict__ child, const int* __restrict__ relmap,
                  const int* __restrict__ a_src, const int* __restrict__ a_pos,
                  const double* __restrict__ Ax, T* __restrict__ Ls, T* __restrict__ Us, int LD,
                  int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const FrontDesc f = fronts[list[blockIdx.x]];
    small_front<T>(f, reinterpret_cast<T*>(smem_raw), LD, threadIdx.x >> 5, blockDim.x >> 5,
                   [] { __syncthreads(); }, fronts, child, relmap, a_src, a_pos, Ax, Ls, Us,
                   status);
}

// Fronts of at most 16 (8) rows: W = 16 (8) lanes per front, two (four) fronts
// per warp, in step with each other: every loop runs to the warp's longest, so
// that the lanes stay together and a shuffle costs a shuffle.  Lane = row, the
// whole row in registers after the assembly in the group's W x (W + 1) slice
// of shared memory.  s < 0: no front for this group.
constexpr int kTinyFrontRows = 32;

template <typename T, int W>
__device__ void tiny_front_group(int s, const FrontDesc* __restrict__ fronts,
                                 const int* __restrict__ child, const int* __restrict__ relmap,
                                 const int* __restrict__ a_src, const int* __restrict__ a_pos,
                                 const double* __restrict__ Ax, T* __restrict__ Ls,
                                 T* __restrict__ Us, int* __restrict__ status, T* Fm) {
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int LD = W + 1, CG = 8;
    const int gl = threadIdx.x & (W - 1);
    FrontDesc f;
    f.m = f.c = f.child_beg = f.child_end = f.a_beg = f.a_end = 0;
    f.uoff = -1;
    if (s >= 0) f = fronts[s];
    const int m = f.m, c = f.c, nch = f.child_end - f.child_beg;
    int src = -1, pos = 0;
    if (f.a_beg + gl < f.a_end) {
        src = a_src[f.a_beg + gl];
        pos = a_pos[f.a_beg + gl];
    }
    int g_id = gl < nch ? child[f.child_beg + gl] : -1;
#pragma unroll
    for (int j = 0; j < W; ++j) Fm[gl + j * LD] = T(0);
    // the children of a batch of up to W, one per lane; the trip at hand: CG
    // columns from j0 on of child h of the batch, maxuc the warp's longest
    const int maxch = __reduce_max_sync(ALL, nch);
    int64_t g_u = 0;
    int g_uc = 0, g_ldu = 0, g_rel = 0;
    int h = 0, nb = 0, j0 = 0, uc = 0, maxuc = 0;
    auto describe = [&]() {
        g_uc = 0;
        if (g_id >= 0) {
            const FrontDesc& g = fronts[g_id];
            g_uc = g.m - g.c;
            g_ldu = g.ldu;
            g_rel = g.rows_off + g.c;
            g_u = g.uoff;
        }
    };
    T v[CG];
    int ri = 0;
    auto fetch = [&]() {  // child h's columns j0 .., rows lane
        if (h >= nb) return;
        if (j0 == 0) {
            uc = __shfl_sync(ALL, g_uc, h, W);
            maxuc = __reduce_max_sync(ALL, uc);
            const int* rm = relmap + __shfl_sync(ALL, g_rel, h, W);
            ri = gl < uc ? rm[gl] : 0;
        }
        const int ldu = __shfl_sync(ALL, g_ldu, h, W);
        const T* U = Us + __shfl_sync(ALL, g_u, h, W);
#pragma unroll
        for (int e = 0; e < CG; ++e) {
            v[e] = T(0);
            if (gl < uc && gl >= j0 + e) v[e] = U[gl + (int64_t)(j0 + e) * ldu];
        }
    };
    describe();
    const T av = src >= 0 ? (T)Ax[src] : T(0);
    nb = min(W, maxch);
    fetch();
    __syncwarp();
    if (src >= 0) Fm[(pos & 0xffff) + (pos >> 16) * LD] = av;
    const int na = __reduce_max_sync(ALL, f.a_end - f.a_beg);
    for (int e0 = W; e0 < na; e0 += W) {
        const int e = f.a_beg + e0 + gl;
        if (e < f.a_end) {
            src = a_src[e];
            if (src >= 0) {
                pos = a_pos[e];
                Fm[(pos & 0xffff) + (pos >> 16) * LD] = (T)Ax[src];
            }
        }
    }
    __syncwarp();
    for (int hb = 0; hb < maxch;) {
        while (h < nb) {
            T w[CG];
#pragma unroll
            for (int e = 0; e < CG; ++e) w[e] = v[e];
            const int cnt = uc, wi = ri, jb = j0;
            j0 += CG;
            if (j0 >= maxuc) ++h, j0 = 0;
            fetch();
            T* at[CG];  // distinct columns: all reads before the writes
#pragma unroll
            for (int e = 0; e < CG; ++e) {
                at[e] = Fm + wi + __shfl_sync(ALL, wi, jb + e, W) * LD;
                if (gl < cnt && gl >= jb + e) w[e] += *at[e];
            }
#pragma unroll
            for (int e = 0; e < CG; ++e)
                if (gl < cnt && gl >= jb + e) *at[e] = w[e];
            __syncwarp();
        }
        hb += W;
        if (hb >= maxch) break;
        h = 0;
        nb = min(W, maxch - hb);
        g_id = hb + gl < nch ? child[f.child_beg + hb + gl] : -1;
        describe();
        fetch();
    }
    T a[W];
#pragma unroll
    for (int j = 0; j < W; ++j) a[j] = Fm[gl + j * LD];
    const int maxc = __reduce_max_sync(ALL, c);
#pragma unroll
    for (int k = 0; k < W; ++k) {
        if (k >= maxc) break;
        const T piv = __shfl_sync(ALL, a[k], k, W);
        T root, inv;
        pivot_root(piv, root, inv);
        if (k < c && gl == k && !(piv > T(0))) flag_pivot(status, f.first_col + k);
        const T l = k < c && gl >= k ? a[k] * inv : T(0);
        if (k < c) a[k] = gl == k ? root : l;
#pragma unroll
        for (int j = k + 1; j < W; ++j) a[j] -= l * __shfl_sync(ALL, l, j, W);
    }
    // (one warp alone issues an instruction every five cycles or so: pointers
    // walked along the columns, and no branch but the loops')
    const int row = gl < m ? gl : -1;
    T* o = Ls + f.loff + gl;
#pragma unroll
    for (int j = 0; j < W; ++j) {
        if (j >= maxc) break;
        if ((j < c) & (row >= 0)) *o = gl >= j ? a[j] : T(0);
        o += f.ldl;
    }
    const int maxm = __reduce_max_sync(ALL, m);
    const int first = f.uoff >= 0 ? c : W;
    o = Us + f.uoff + (gl - c) - (int64_t)c * f.ldu;
#pragma unroll
    for (int j = 0; j < W; ++j) {
        if (j >= maxm) break;
        if ((j >= first) & (j <= row)) *o = a[j];
        o += f.ldu;
    }
    __syncwarp();  // the slice is reused by the group's next front
}

// One level's fronts of at most 32 rows as warp tasks over a rows-descending
// list: tasks [0, n32) one front each (17..32 rows), then two fronts of 9..16
// rows per task, then four of at most 8; persistent warps take tasks with
// the grid's warp count as stride.
template <typename T>
__global__ void __launch_bounds__(128)
    k_tiny_fronts(const FrontDesc* __restrict__ fronts, const int* __restrict__ list, int n32,
                  int n16, int n8, const int* __restrict__ child, const int* __restrict__ relmap,
                  const int* __restrict__ a_src, const int* __restrict__ a_pos,
                  const double* __restrict__ Ax, T* __restrict__ Ls, T* __restrict__ Us,
                  int* __restrict__ status) {
    constexpr int LD = small_ld<T>(kTinyFrontRows);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    T* slice = reinterpret_cast<T*>(smem_raw) + (size_t)warp * kTinyFrontRows * LD;
    const int t16 = (n16 + 1) / 2, t8 = (n8 + 3) / 4, ntask = n32 + t16 + t8;
    for (int t = blockIdx.x * wpb + warp; t < ntask; t += gridDim.x * wpb) {
        if (t < n32) {
            const FrontDesc f = fronts[list[t]];
            small_front<T>(f, slice, LD, 0, 1, [] { __syncwarp(); }, fronts, child, relmap, a_src,
                           a_pos, Ax, Ls, Us, status);
        } else if (t < n32 + t16) {
            const int k = 2 * (t - n32) + (lane >> 4);
            tiny_front_group<T, 16>(k < n16 ? list[n32 + k] : -1, fronts, child, relmap, a_src,
                                    a_pos, Ax, Ls, Us, status, slice + (lane >> 4) * 16 * 17);
        } else {
            const int k = 4 * (t - n32 - t16) + (lane >> 3);
            tiny_front_group<T, 8>(k < n8 ? list[n32 + n16 + k] : -1, fronts, child, relmap, a_src,
                                   a_pos, Ax, Ls, Us, status, slice + (lane >> 3) * 8 * 9);
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// large fronts: assembly
// ---------------------------------------------------------------------------

template <typename T>
__global__ void __launch_bounds__(256)
    k_big_assemble(const FrontDesc* __restrict__ fronts, const int* __restrict__ items,
                   const int* __restrict__ before, int nitems, int CB,
                   const int* __restrict__ child, const int* __restrict__ relmap,
                   const int* __restrict__ a_src, const int* __restrict__ a_pos,
                   const int* __restrict__ a_colptr, const int* __restrict__ a_colptr_off,
                   const int* __restrict__ asm_off, const int* __restrict__ asm_range,
                   const double* __restrict__ Ax, T* __restrict__ Ls, T* __restrict__ Us) {
    extern __shared__ int rel_sh[];  // a child's relative map from its first column in range
    const int it = find_item(before, nitems, blockIdx.x);
    const int s = items[it];
    const int blk = blockIdx.x - before[it];
    const FrontDesc f = fronts[s];
    const int j0 = blk * CB, j1 = min(j0 + CB, f.m);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int nch = f.child_end - f.child_beg;
    const int* ranges = asm_range + asm_off[s] + blk * nch * 2;

    for (int jj = j0; jj < j1; ++jj) {
        if (jj < f.c) {
            T* col = Ls + f.loff + (int64_t)jj * f.ldl;
            for (int r = tid; r < f.m; r += nt) col[r] = T(0);
        } else {
            T* col = Us + f.uoff + (int64_t)(jj - f.c) * f.ldu;
            for (int r = jj - f.c + tid; r < f.m - f.c; r += nt) col[r] = T(0);
        }
    }
    __syncthreads();
    if (j0 < f.c) {
        const int* cp = a_colptr + a_colptr_off[s];
        int e0 = f.a_beg + cp[j0], e1 = f.a_beg + cp[min(j1, f.c)];
        for (int e = e0 + tid; e < e1; e += nt) {
            int src = a_src[e];
            if (src >= 0) {
                int pos = a_pos[e];
                Ls[f.loff + (pos & 0xffff) + (int64_t)(pos >> 16) * f.ldl] = (T)Ax[src];
            }
        }
    }
    __syncthreads();
    // children one after another (deterministic sums); each child's update
    // columns that land in [j0, j1) were located on the host.  The child's
    // relative map goes to shared memory and every thread keeps four
    // independent loads in flight before its read-modify-writes.
    for (int h = 0; h < nch; ++h) {
        const int jlo = ranges[2 * h], jhi = ranges[2 * h + 1];
        if (jlo == jhi) continue;
        const FrontDesc g = fronts[child[f.child_beg + h]];
        const int uc = g.m - g.c;
        const int* rm = relmap + g.rows_off + g.c;
        for (int q = jlo + tid; q < uc; q += nt) rel_sh[q - jlo] = rm[q];
        __syncthreads();
        const T* U = Us + g.uoff;
        for (int jc = jlo; jc < jhi; ++jc) {
            const int pc = rel_sh[jc - jlo];
            const T* ucol = U + (int64_t)jc * g.ldu;
            for (int ic0 = jc + tid; ic0 < uc; ic0 += 4 * nt) {
                T v[4];
                int pr[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int ic = ic0 + u * nt;
                    pr[u] = ic < uc ? rel_sh[ic - jlo] : -1;
                    v[u] = ic < uc ? ucol[ic] : T(0);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (pr[u] >= 0) *front_elem(Ls, Us, f, pr[u], pc) += v[u];
            }
        }
        __syncthreads();
    }
}

// Warp-per-column variant: no block barriers but the one behind the table of
// the block's children.  Each warp builds its column in windows of W rows (W a
// multiple of 16) in its own shared slice, so the slice does not grow with the
// front.  A child's columns landing in the CTA's block of CB columns are at most
// CB (the relative map is injective); which of them lands in which column, and
// where the child's values are, sits in the table for fronts of up to 32
// children (others look it up per column, by one ballot over the child's
// range).  The child rows landing in a window are one contiguous range
// (increasing relative map), read from the per-16-row block table asm_range where
// the window is not the whole column.  Every front entry gets its A value (or
// zero), then the children's contributions in child order: the sums of a
// child-by-child extend-add.  The next 256 values of the children are under way
// while the last are added.  Bound by instruction issue (two slots of three taken
// at 0.95 TB/s on fronts of a few hundred rows), so neither two columns per
// warp nor fewer values per trip gained: 48^3 FP64 2.10 -> 1.93 ms, 64^3 FP32
// 3.72 -> 3.60 against the lookup per column with no load ahead.
template <typename T>
__global__ void __launch_bounds__(256)
    k_big_assemble_warp(const FrontDesc* __restrict__ fronts, const int* __restrict__ items,
                        const int* __restrict__ before, int nitems, int CB,
                        const int* __restrict__ child, const int* __restrict__ relmap,
                        const int* __restrict__ a_src, const int* __restrict__ a_pos,
                        const int* __restrict__ a_colptr, const int* __restrict__ a_colptr_off,
                        const int* __restrict__ asm_off, const int* __restrict__ asm_range,
                        const double* __restrict__ Ax, T* __restrict__ Ls, T* __restrict__ Us,
                        int W) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int KIDS = 32, NL = 8;
    // the block's children: update matrix, row map, and per column of the
    // block the child's column that lands there (-1: none)
    __shared__ int64_t s_u[KIDS];
    __shared__ int s_rm[KIDS], s_ldu[KIDS], s_uc[KIDS];
    __shared__ int s_jc[KIDS][kAssembleCols];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    T* colbuf = reinterpret_cast<T*>(smem_raw) + (size_t)warp * W;
    const int it = find_item(before, nitems, blockIdx.x);
    const int s = items[it];
    const int blk = blockIdx.x - before[it];
    const FrontDesc f = fronts[s];
    const int j0 = blk * CB, j1 = min(j0 + CB, f.m);
    const int nch = f.child_end - f.child_beg;
    const int* rtab = asm_range + asm_off[s];  // [16-row block][child] -> [lo, hi)
    const int* ranges = rtab + blk * nch * 2;
    const int* cp = j0 < f.c ? a_colptr + a_colptr_off[s] : nullptr;
    const bool table = nch <= KIDS;
    if (table) {
        for (int h = warp; h < nch; h += nw) {
            const FrontDesc& g = fronts[child[f.child_beg + h]];
            const int jlo = ranges[2 * h], jhi = ranges[2 * h + 1];
            if (lane < kAssembleCols) s_jc[h][lane] = -1;
            if (lane == 0) {
                s_u[h] = g.uoff;
                s_ldu[h] = g.ldu;
                s_uc[h] = g.m - g.c;
                s_rm[h] = g.rows_off + g.c;
            }
            __syncwarp();
            if (jlo + lane < jhi)
                s_jc[h][__ldg(relmap + g.rows_off + g.c + jlo + lane) - j0] = jlo + lane;
        }
        __syncthreads();
    }
    for (int jj = j0 + warp; jj < j1; jj += nw) {
        const bool inL = jj < f.c;
        const int rlo = inL ? 0 : jj;
        for (int R0 = (rlo / W) * W; R0 < f.m; R0 += W) {
            const int R1 = min(R0 + W, f.m), w0 = max(R0, rlo);
            const int b0 = R0 / 16, b1 = (R1 - 1) / 16;
            // the trip at hand: NL x 32 of child h's rows >= its column, from
            // ic0 on; h == nch at the end.  One trip's loads are under way while
            // the one before is added.
            int h = -1, ic0 = 0, ihi = 0;
            const int* rm = nullptr;
            const T* ucol = nullptr;
            auto settle = [&]() {
                while (ic0 >= ihi) {
                    if (++h >= nch) return;
                    int jc = -1, uc = 0;
                    if (table) {
                        jc = s_jc[h][jj - j0];
                        if (jc < 0) continue;
                        uc = s_uc[h];
                        rm = relmap + s_rm[h];
                        ucol = Us + s_u[h] + (int64_t)jc * s_ldu[h];
                    } else {
                        const int jlo = ranges[2 * h], jhi = ranges[2 * h + 1];
                        if (jlo == jhi) continue;
                        const FrontDesc& g = fronts[child[f.child_beg + h]];
                        rm = relmap + g.rows_off + g.c;
                        const int cand = jlo + lane;
                        const unsigned hit =
                            __ballot_sync(ALL, cand < jhi && __ldg(rm + cand) == jj);
                        if (!hit) continue;
                        jc = jlo + __ffs(hit) - 1;
                        uc = g.m - g.c;
                        ucol = Us + g.uoff + (int64_t)jc * g.ldu;
                    }
                    // child rows >= jc landing in rows [R0, R1) of the parent
                    ic0 = R0 <= jj ? jc : max(jc, rtab[(b0 * nch + h) * 2]);
                    ihi = R1 == f.m ? uc : rtab[(b1 * nch + h) * 2 + 1];
                }
            };
            int pr[NL];
            T v[NL];
            auto fetch = [&]() {
                if (h >= nch) return;
#pragma unroll
                for (int u = 0; u < NL; ++u) {
                    const int ic = ic0 + lane + u * 32;
                    pr[u] = ic < ihi ? __ldg(rm + ic) : -1;
                    v[u] = ic < ihi ? __ldg(ucol + ic) : T(0);
                }
            };
            settle();
            fetch();
            for (int r = w0 + lane; r < R1; r += 32) colbuf[r - R0] = T(0);
            __syncwarp();
            if (inL) {
                const int e0 = f.a_beg + cp[jj], e1 = f.a_beg + cp[jj + 1];
                for (int e = e0 + lane; e < e1; e += 32) {
                    const int src = a_src[e], row = a_pos[e] & 0xffff;
                    if (src >= 0 && row >= R0 && row < R1) colbuf[row - R0] = (T)Ax[src];
                }
                __syncwarp();
            }
            while (h < nch) {  // children in order
                int q[NL];
                T x[NL];
#pragma unroll
                for (int u = 0; u < NL; ++u) q[u] = pr[u] - R0, x[u] = v[u];
                ic0 += NL * 32;
                settle();
                fetch();
                // distinct rows: all reads before the writes
#pragma unroll
                for (int u = 0; u < NL; ++u)
                    if (q[u] + R0 >= 0) x[u] += colbuf[q[u]];
#pragma unroll
                for (int u = 0; u < NL; ++u)
                    if (q[u] + R0 >= 0) colbuf[q[u]] = x[u];
                __syncwarp();
            }
            if (inL) {
                T* col = Ls + f.loff + (int64_t)jj * f.ldl;
                for (int r = w0 + lane; r < R1; r += 32) col[r] = colbuf[r - R0];
            } else {
                T* col = Us + f.uoff + (int64_t)(jj - f.c) * f.ldu;
                for (int r = w0 + lane; r < R1; r += 32) col[r - f.c] = colbuf[r - R0];
            }
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------------------
// large fronts: tiles
// ---------------------------------------------------------------------------

// Factor diagonal tile k of front f in place and store its inverse (TB x TB,
// column-major, zero above the diagonal) at Dk (potrf_tile_core on a copy in
// shared memory; a partial tile (n < 64) is padded with the identity).
// S, W: TB x kPotrfLD.
template <typename T, int TB>
__device__ void potrf_diag_tile(const FrontDesc& f, int k, T* Ls, T* Dk, T* S, T* W,
                                int* status) {
    constexpr int LD = kPotrfLD;
    const int tid = threadIdx.x, nt = blockDim.x;
    const TileRange tk = tile_range(k, f.m, f.c, TB);
    const int n = tk.size;
    T* base = Ls + f.loff + tk.start + (int64_t)tk.start * f.ldl;
    for (int idx = tid; idx < TB * TB; idx += nt) {
        int j = idx / TB, i = idx - j * TB;
        T v = (i == j) ? T(1) : T(0);
        if (i < n && j < n && i >= j) v = base[i + (int64_t)j * f.ldl];
        S[i + j * LD] = v;
    }
    potrf_tile_core<T, TB>(S, W, n, f.first_col + tk.start, status);
    for (int idx = tid; idx < TB * TB; idx += nt) {
        int j = idx / TB, i = idx - j * TB;
        if (i < n && j < n && i >= j) base[i + (int64_t)j * f.ldl] = S[i + j * LD];
        Dk[idx] = (i >= j && i < n && j < n) ? W[i + j * LD] : T(0);
    }
}

template <typename T, int TB>
__global__ void __launch_bounds__(256)
    k_tile_potrf(const FrontDesc* __restrict__ fronts, const int* __restrict__ list, int k,
                 const int64_t* __restrict__ dinv_off, T* __restrict__ Ls, T* __restrict__ Dinv,
                 int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* S = reinterpret_cast<T*>(smem_raw);
    T* W = S + TB * kPotrfLD;
    const int s = list[blockIdx.x];
    const FrontDesc f = fronts[s];
    if (k >= tiles_l(f.c, TB)) return;
    potrf_diag_tile<T, TB>(f, k, Ls, Dinv + dinv_off[s] + (int64_t)k * TB * TB, S, W, status);
}

// X = A_ik inv(L_kk)' in place, CTA per row tile below the panel tile.
template <typename T, int TB>
__global__ void __launch_bounds__(256)
    k_tile_trsm(const FrontDesc* __restrict__ fronts, const int* __restrict__ items,
                const int* __restrict__ before, int nitems, int k,
                const int64_t* __restrict__ dinv_off, T* __restrict__ Ls,
                const T* __restrict__ Dinv) {
    static_assert(TB == 64, "4x4 register tile over 256 threads assumes TB = 64");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* As = reinterpret_cast<T*>(smem_raw);  // [K][TB]
    T* Bs = As + TB * TB;                    // [K][TB]: inv(L_kk)' columns
    const int it = find_item(before, nitems, blockIdx.x);
    const int s = items[it];
    const FrontDesc f = fronts[s];
    const int i = k + 1 + (blockIdx.x - before[it]);
    const TileRange tk = tile_range(k, f.m, f.c, TB);
    const TileRange ti = tile_range(i, f.m, f.c, TB);
    const int tid = threadIdx.x;
    const int K = tk.size;
    T* aik = Ls + f.loff + ti.start + (int64_t)tk.start * f.ldl;
    const T* Dk = Dinv + dinv_off[s] + (int64_t)k * TB * TB;  // inv(L_kk), col-major TB
    for (int idx = tid; idx < TB * K; idx += 256) {
        int q = idx / TB, r = idx - q * TB;
        As[q * TB + r] = r < ti.size ? aik[r + (int64_t)q * f.ldl] : T(0);
        Bs[q * TB + r] = Dk[r + q * TB];  // Bs[q][j] = inv(L)[j][q]
    }
    __syncthreads();
    T acc[4][4];
    tile_gemm_nt_acc<T, TB>(As, Bs, K, acc);
    const int r0 = (tid & 15) * 4, c0 = (tid >> 4) * 4;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        int cc = c0 + b;
        if (cc >= K) continue;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            int rr = r0 + a;
            if (rr < ti.size) aik[rr + (int64_t)cc * f.ldl] = acc[a][b];
        }
    }
}

// jcap < 0: every lower tile right of panel tile k (the FP64 schedule).
// jcap >= 0: only tile columns k < j <= jcap (the rest of a 256-column panel;
// the trailing part then gets one tensor-core update per panel).
template <typename T, int TB>
__global__ void __launch_bounds__(256)
    k_tile_update(const FrontDesc* __restrict__ fronts, const int* __restrict__ items,
                  const int* __restrict__ before, int nitems, int k, int jcap,
                  const int64_t* __restrict__ dinv_off, T* __restrict__ Ls, T* __restrict__ Us,
                  T* __restrict__ Dinv, int* __restrict__ status) {
    static_assert(TB == 64, "4x4 register tile over 256 threads assumes TB = 64");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* As = reinterpret_cast<T*>(smem_raw);  // [K][TB]
    T* Bs = As + TB * TB;                    // [K][TB]
    const int it = find_item(before, nitems, blockIdx.x);
    const int s = items[it];
    const FrontDesc f = fronts[s];
    int i, j;
    if (jcap < 0) {
        int ii, jj;
        lower_index(blockIdx.x - before[it], ii, jj);
        i = k + 1 + ii;
        j = k + 1 + jj;
    } else {  // column-major over the panel's remaining tile columns
        const int NT = tiles_l(f.c, TB) + (f.m - f.c + TB - 1) / TB;
        int l = blockIdx.x - before[it];
        j = k + 1;
        while (l >= NT - j) {
            l -= NT - j;
            ++j;
        }
        i = j + l;
    }
    const TileRange tk = tile_range(k, f.m, f.c, TB);
    const TileRange ti = tile_range(i, f.m, f.c, TB);
    const TileRange tj = tile_range(j, f.m, f.c, TB);
    const int tid = threadIdx.x;
    const int K = tk.size;
    const T* pa = Ls + f.loff + ti.start + (int64_t)tk.start * f.ldl;
    const T* pb = Ls + f.loff + tj.start + (int64_t)tk.start * f.ldl;
    for (int idx = tid; idx < TB * K; idx += 256) {
        int q = idx / TB, r = idx - q * TB;
        As[q * TB + r] = r < ti.size ? pa[r + (int64_t)q * f.ldl] : T(0);
        Bs[q * TB + r] = r < tj.size ? pb[r + (int64_t)q * f.ldl] : T(0);
    }
    __syncthreads();
    T acc[4][4];
    tile_gemm_nt_acc<T, TB>(As, Bs, K, acc);
    const int r0 = (tid & 15) * 4, c0 = (tid >> 4) * 4;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        int cc = c0 + b;
        if (cc >= tj.size) continue;
        int gc = tj.start + cc;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            int rr = r0 + a;
            if (rr >= ti.size) continue;
            int gr = ti.start + rr;
            if (gr < gc) continue;
            *front_elem(Ls, Us, f, gr, gc) -= acc[a][b];
        }
    }
    // the next diagonal tile is final now: factor it for the next step
    if (i == k + 1 && j == k + 1 && i < tiles_l(f.c, TB) && (jcap < 0 || i <= jcap)) {
        __syncthreads();
        potrf_diag_tile<T, TB>(f, i, Ls, Dinv + dinv_off[s] + (int64_t)i * TB * TB, As,
                               As + TB * kPotrfLD, status);
    }
}

// Columns c0 .. of L into compressed columns, a warp per column.
template <typename T>
__global__ void __launch_bounds__(256)
    k_pack_columns(const FrontDesc* __restrict__ fronts, const int* __restrict__ col_front,
                   const int64_t* __restrict__ Lp, const T* __restrict__ Ls, int c0, int c1,
                   double* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    for (int col = c0 + (int)(blockIdx.x * 8 + (threadIdx.x >> 5)); col < c1;
         col += gridDim.x * 8) {
        const FrontDesc& f = fronts[col_front[col]];
        const int j = col - f.first_col, m = f.m;
        const T* src = Ls + f.loff + (int64_t)j * f.ldl;
        double* dst = out + (Lp[col] - Lp[c0]) - j;
        for (int i = j + lane; i < m; i += 32) dst[i] = (double)src[i];
    }
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------

// rows per window of the warp-per-column assembly's column buffers
constexpr int kAssembleWindow = 1024;
constexpr size_t kAssembleColsSmemMax = 8 * kAssembleWindow * sizeof(double);

// shared memory of the tile kernels: two 64 x kPotrfLD buffers (operands of
// the tile products in 64 x 65 of them, or S and W of the diagonal-tile
// factorization)
template <typename T>
static size_t diag_smem() {
    return (size_t)2 * kTile * kPotrfLD * sizeof(T);
}

// The level's small fronts in pieces, piece i on sts[i]: the tiny fronts
// (piece 0), then one k_small_front launch per size bucket.
template <typename T>
void launch_small_fronts(const DevPlan& D, int level, T* Ls, T* Us, const double* Ax,
                         int* status, const cudaStream_t* sts) {
    {  // fronts of at most 32 rows (the first two buckets): one, two or four per warp
        const int beg = D.h_small_ptr[level * kSmallBuckets];
        const int end = D.h_small_ptr[level * kSmallBuckets + Plan::kTinyBuckets];
        const cudaStream_t st = sts[0];
        if (end > beg) {
            double by = 0;
            for (int b = 0; b < Plan::kTinyBuckets; ++b)
                by += D.h_small_bytes[level * kSmallBuckets + b];
            ProfScope ps(D.prof, KC_SMALL_FRONT, st, 0, by * sizeof(T) / 8.0);
            const size_t smem = (size_t)4 * kTinyFrontRows * small_ld<T>(kTinyFrontRows) * sizeof(T);
            // the level's slice of the rows-descending warp list: its fronts
            // of 17..32 rows end the part above 16 rows, then 9..16, then <= 8
            const int* cnt = D.solve.warp_cnt.data() + 3 * level;
            const int n32 = D.h_small_ptr[level * kSmallBuckets + 2] -
                            D.h_small_ptr[level * kSmallBuckets + 1];
            const int n16 = cnt[1], n8 = cnt[2];
            const int ntask = n32 + (n16 + 1) / 2 + (n8 + 3) / 4;
            const int blocks = std::min((ntask + 3) / 4, D.tiny_blocks_cap);
            // a few fronts of 17..32 rows alone: four warps each (a warp each
            // leaves the GPU idle; 24 x 23 grid: 8.5 -> 5.9 us a level, a root of 29
            // columns 21 -> 13.5)
            if (n16 + n8 == 0 && n32 <= 2 * (D.num_sms > 0 ? D.num_sms : 148))
                k_small_front<T><<<n32, 128, smem / 4, st>>>(
                    D.fronts, D.solve.warp_list + beg + (cnt[0] - n32), D.child, D.relmap, D.a_src,
                    D.a_pos, Ax, Ls, Us, small_ld<T>(kTinyFrontRows), status);
            else
                k_tiny_fronts<T><<<blocks, 128, smem, st>>>(
                    D.fronts, D.solve.warp_list + beg + (cnt[0] - n32), n32, n16, n8, D.child,
                    D.relmap, D.a_src, D.a_pos, Ax, Ls, Us, status);
        }
    }
    for (int b = Plan::kTinyBuckets; b < kSmallBuckets; ++b) {
        int beg = D.h_small_ptr[level * kSmallBuckets + b];
        int end = D.h_small_ptr[level * kSmallBuckets + b + 1];
        if (end == beg) continue;
        int MB = Plan::small_limit[b];
        int LD = small_ld<T>(MB);
        size_t smem = (size_t)MB * LD * sizeof(T);
        const int threads = D.small_threads[b];
        const cudaStream_t st = sts[1 + b - Plan::kTinyBuckets];
        ProfScope ps(D.prof, KC_SMALL_FRONT, st, 0,
                     D.h_small_bytes[level * kSmallBuckets + b] * sizeof(T) / 8.0);
        k_small_front<T><<<end - beg, threads, smem, st>>>(D.fronts, D.small_list + beg, D.child,
                                                          D.relmap, D.a_src, D.a_pos, Ax, Ls, Us,
                                                          LD, status);
    }
}

template <typename T>
void launch_large_level(const DevPlan& D, int level, T* Ls, T* Us, T* Dinv, const double* Ax,
                        int* status, cudaStream_t st) {
    const int lb = D.h_large_ptr[level], le = D.h_large_ptr[level + 1];
    if (le == lb) return;
    const DevSchedule& S = D.sched64;
    const WorkList& asl = D.h_assemble[level];
    {
        ProfScope ps(D.prof, KC_ASSEMBLE, st);
        k_big_assemble<T><<<asl.nctas, 256, D.max_u * sizeof(int), st>>>(
            D.fronts, S.items + asl.off, S.before + asl.off, asl.nitems, kAssembleCols, D.child,
            D.relmap, D.a_src, D.a_pos, D.a_colptr, D.a_colptr_off, D.asm_off, D.asm_range, Ax,
            Ls, Us);
    }
    {
        ProfScope ps(D.prof, KC_POTRF, st);
        k_tile_potrf<T, kTile><<<le - lb, 256, diag_smem<T>(), st>>>(D.fronts, D.large_list + lb,
                                                                     0, D.dinv_off, Ls, Dinv,
                                                                     status);
    }
    const size_t gsm = diag_smem<T>();
    for (int q = S.h_level_beg[level]; q < S.h_level_beg[level + 1]; ++q) {
        const WorkList& tr = S.h_trsm[q];
        const WorkList& up = S.h_update[q];
        if (tr.nctas > 0) {
            ProfScope ps(D.prof, KC_TRSM, st);
            k_tile_trsm<T, kTile><<<tr.nctas, 256, gsm, st>>>(
                D.fronts, S.items + tr.off, S.before + tr.off, tr.nitems, tr.step, D.dinv_off, Ls,
                Dinv);
        }
        if (up.nctas > 0) {
            ProfScope ps(D.prof, KC_SCHUR, st, D.h_update_flops[q]);
            k_tile_update<T, kTile><<<up.nctas, 256, gsm, st>>>(
                D.fronts, S.items + up.off, S.before + up.off, up.nitems, up.step, -1, D.dinv_off,
                Ls, Us, Dinv, status);
        }
    }
}

// Large fronts in 256-column panels: per panel one launch of dependency-
// ordered row-tile tasks (k_panel: diagonal tiles, triangular solves and the
// panel's own updates), then one wide Schur update of the whole trailing
// part -- tcgen05 tensor cores (TF32) for FP32, the FP64 matrix instructions
// for FP64.  status[1] receives a device wait's error code (1, 2:
// the tensor-core pipeline; 3: a panel dependency wait; 4: a panel ticket
// counter not cleared).
template <typename T>
static void launch_large_level_panels(const DevPlan& D, int level, T* Ls, T* Us, T* Dinv,
                                      const double* Ax, int* status, int smode,
                                      cudaStream_t st) {
    const DevSchedule& S = D.psched;
    const size_t gsm = diag_smem<T>();
    for (int q = S.h_op_beg[level]; q < S.h_op_beg[level + 1]; ++q) {
        const PanelOp& op = S.h_ops[q];
        const WorkList& w = op.w;
        if (op.kind == OP_PANEL ? op.ntasks == 0 : w.nctas == 0) continue;
        switch (op.kind) {
            case OP_ASSEMBLE: {
                ProfScope ps(D.prof, KC_ASSEMBLE, st, 0, op.elems * sizeof(T) + op.xbytes);
                // a warp per column, 8 warps, columns built in windows of
                // kAssembleWindow rows (the whole column when shorter)
                const int W = std::min(kAssembleWindow, (D.h_level_max_m[level] + 15) & ~15);
                k_big_assemble_warp<T><<<w.nctas, 256, (size_t)8 * W * sizeof(T), st>>>(
                    D.fronts, S.items + w.off, S.before + w.off, w.nitems, kAssembleCols, D.child,
                    D.relmap, D.a_src, D.a_pos, D.a_colptr, D.a_colptr_off, D.asm_off,
                    D.asm_range, Ax, Ls, Us, W);
                break;
            }
            case OP_POTRF: {
                ProfScope ps(D.prof, KC_POTRF, st, op.flops, op.elems * sizeof(T));
                k_tile_potrf<T, kTile><<<w.nitems, 256, diag_smem<T>(), st>>>(
                    D.fronts, S.items + w.off, op.arg, D.dinv_off, Ls, Dinv, status);
                break;
            }
            case OP_TRSM: {
                ProfScope ps(D.prof, KC_TRSM, st, op.flops, op.elems * sizeof(T));
                k_tile_trsm<T, kTile><<<w.nctas, 256, gsm, st>>>(
                    D.fronts, S.items + w.off, S.before + w.off, w.nitems, op.arg, D.dinv_off, Ls,
                    Dinv);
                break;
            }
            case OP_UPDATE_PANEL: {
                ProfScope ps(D.prof, KC_TRSM, st, op.flops, op.elems * sizeof(T));
                k_tile_update<T, kTile><<<w.nctas, 256, gsm, st>>>(
                    D.fronts, S.items + w.off, S.before + w.off, w.nitems, op.arg, op.arg2,
                    D.dinv_off, Ls, Us, Dinv, status);
                break;
            }
            case OP_PANEL: {
                ProfScope ps(D.prof, KC_TRSM, st, op.flops, op.elems * sizeof(T));
                // the panel scratch the tensor-core Schur update reads:
                // the 3xTF32 hi/lo split (1) or the BF16 copy (2)
                launch_panel<T>(D, op, Ls, Dinv, status,
                                sizeof(T) == 4 ? (smode == kSchurBF16 ? 2 : 1) : 0, st);
                break;
            }
            case OP_SCHUR_TC: {
                // one update per panel: the FP64 factor's (the tensor-core
                // path runs the deferred updates below instead)
                if constexpr (sizeof(T) == 8) {
                    ProfScope ps(D.prof, KC_SCHUR, st, op.flops, op.elems * sizeof(T));
                    launch_schur_f64(D, w, op.arg, kPanel, Ls, Us, st);
                }
                break;
            }
            case OP_SCHUR_NEXT:
            case OP_SCHUR_REST: {
                if constexpr (sizeof(T) == 4) {
                    ProfScope ps(D.prof, KC_SCHUR, st, op.flops, op.elems * sizeof(T));
                    launch_schur_tc(D, w, op.arg, kPanel, op.arg2, op.kind == OP_SCHUR_NEXT, Ls,
                                    Us, status + 1, smode, st);
                }
                break;
            }
        }
    }
}

template <typename T>
void pack_columns(const DevPlan& D, const T* Ls, int c0, int c1, double* out, cudaStream_t st) {
    const int sms = D.num_sms > 0 ? D.num_sms : 148;
    k_pack_columns<T><<<std::min((c1 - c0 + 7) / 8, 8 * sms), 256, 0, st>>>(
        D.fronts, D.adj.col_front, D.adj.Lp, Ls, c0, c1, out);
}
template void pack_columns<double>(const DevPlan&, const double*, int, int, double*,
                                   cudaStream_t);
template void pack_columns<float>(const DevPlan&, const float*, int, int, double*, cudaStream_t);

template <typename T>
static void set_factor_attributes() {
    cudaFuncSetAttribute(k_small_front<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         227 * 1024);
    cudaFuncSetAttribute(k_tile_update<T, kTile>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)diag_smem<T>());
    cudaFuncSetAttribute(k_tile_trsm<T, kTile>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)diag_smem<T>());
    cudaFuncSetAttribute(k_tile_potrf<T, kTile>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)diag_smem<T>());
    cudaFuncSetAttribute(k_big_assemble<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         227 * 1024);
    cudaFuncSetAttribute(k_big_assemble_warp<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kAssembleColsSmemMax);
}

void init_factor_kernels() {
    set_factor_attributes<double>();
    set_factor_attributes<float>();
}

// Level by level.  A level's small and large fronts depend only on lower
// levels, so its small fronts run beside its large fronts, each piece (the
// tiny fronts, each k_small_front size bucket) on a stream of its own (fork
// and join by events; inside a stream capture these become parallel graph
// branches).  Serial while the profiler records, so each class keeps its own
// time.
template <typename T>
void factor_levels(const DevPlan& D, T* Ls, T* Us, T* Dinv, const double* Ax, int* status,
                   cudaStream_t st, int smode) {
    const bool fork = D.fork_ev && !(D.prof && D.prof->on);
    if (D.fsync && D.nfsync > 0) cudaMemsetAsync(D.fsync, 0, (size_t)D.nfsync * sizeof(int), st);
    for (int l = 0; l < D.nlevels; ++l) {
        const bool has_small =
            D.h_small_ptr[(l + 1) * kSmallBuckets] > D.h_small_ptr[l * kSmallBuckets];
        const bool has_large = D.h_large_ptr[l + 1] > D.h_large_ptr[l];
        // pieces of the level's small fronts that have fronts
        bool piece[DevPlan::kSmallPieces];
        int npieces = 0;
        piece[0] = D.h_small_ptr[l * kSmallBuckets + Plan::kTinyBuckets] >
                   D.h_small_ptr[l * kSmallBuckets];
        for (int b = Plan::kTinyBuckets; b < kSmallBuckets; ++b)
            piece[1 + b - Plan::kTinyBuckets] =
                D.h_small_ptr[l * kSmallBuckets + b + 1] > D.h_small_ptr[l * kSmallBuckets + b];
        for (int i = 0; i < DevPlan::kSmallPieces; ++i) npieces += piece[i];
        const bool par = fork && D.piece_st[0] && has_small && (has_large || npieces > 1);
        if (par) {
            // every piece on its own stream beside the large fronts
            cudaEventRecord(D.fork_ev, st);
            for (int i = 0; i < DevPlan::kSmallPieces; ++i)
                if (piece[i]) cudaStreamWaitEvent(D.piece_st[i], D.fork_ev, 0);
            launch_small_fronts<T>(D, l, Ls, Us, Ax, status, D.piece_st);
            for (int i = 0; i < DevPlan::kSmallPieces; ++i)
                if (piece[i]) cudaEventRecord(D.piece_join[i], D.piece_st[i]);
        } else {
            cudaStream_t serial[DevPlan::kSmallPieces];
            for (int i = 0; i < DevPlan::kSmallPieces; ++i) serial[i] = st;
            launch_small_fronts<T>(D, l, Ls, Us, Ax, status, serial);
        }
        // FP32 needs the TMA descriptors of the tensor-core path; without them
        // (descriptor encoding unavailable) it keeps the 64-wide tile schedule
        if (sizeof(T) == 8 || (smode == kSchurBF16 ? D.tmaps_bf16 != nullptr : D.tmaps != nullptr))
            launch_large_level_panels<T>(D, l, Ls, Us, Dinv, Ax, status, smode, st);
        else
            launch_large_level<T>(D, l, Ls, Us, Dinv, Ax, status, st);
        if (par)
            for (int i = 0; i < DevPlan::kSmallPieces; ++i)
                if (piece[i]) cudaStreamWaitEvent(st, D.piece_join[i], 0);
    }
}

template void factor_levels<double>(const DevPlan&, double*, double*, double*, const double*,
                                    int*, cudaStream_t, int);
template void factor_levels<float>(const DevPlan&, float*, float*, float*, const double*, int*,
                                   cudaStream_t, int);

}  // namespace mdgpu
