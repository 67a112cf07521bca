// Selected inverse and the adjoint of logdet A + b' A^-1 b.
//
// For A = L L' (the FP64 factor), Z = A^-1 on the pattern of L satisfies the
// Takahashi recurrence, column by column from the last: with R the rows
// below the diagonal of column j (a clique of the filled graph),
//     y = L(R, j) / L(j, j),   Z(R, j) = -Z(R, R) y,
//     Z(j, j) = 1 / L(j, j)^2 - y' Z(R, j).
// Per front, with its pivot columns in blocks K of NB columns from the last
// and R the front rows below the block, the same in block form:
//     W = inv(L_KK),  Y = L_RK W,  Z_RK = -Z_RR Y,  Z_KK = W'W - Y' Z_RK.
// Z_RR lies inside the front: its pivot part was computed by the later
// blocks, its update part Z_UU is the parent front's Z on the front's update
// rows (gathered through the relative map -- the transpose of the
// extend-add).  So the fronts are processed level by level from the root:
// small fronts a CTA or a warp each (blocks of 8 columns), large fronts in blocks
// of 64 columns over many CTAs per front (below); Z of the pivot columns goes to
// a store laid out like the L panels, Z_UU to the selected inverse's own
// update store.
//
// The gradient of loss = logdet A + b' A^-1 b with respect to the caller's
// lower-triangle values: with x = A^-1 b, d loss / d A = Z - x x' (symmetric),
// so an off-diagonal entry (one value standing for A(i,j) and A(j,i)) gets
// 2 (Z(i,j) - x_i x_j) and a diagonal entry Z(i,i) - x_i^2.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device_common.cuh"
#include "kernels.hpp"
#include "tile64.cuh"

namespace mdgpu {

// Z(r, col), r >= col, front-local indices of front f
// (Z's update part of front f at zoff in the Zu store)
__device__ __forceinline__ double& zelem(double* Zs, double* Zu, const FrontDesc& f,
                                         int64_t zoff, int r, int col) {
    if (col < f.c) return Zs[f.loff + r + (int64_t)col * f.ldl];
    return Zu[zoff + (r - f.c) + (int64_t)(col - f.c) * f.ldu];
}

// Small fronts, the recurrence in blocks of eight pivot columns with the whole
// symmetric Z of the front in shared memory: most have one to a few pivot
// columns, so the gather of Z_UU from the parent is most of the work -- a warp
// takes eight of its columns at a time, lane = row, all loads before the
// stores.  Y = L_RK inv(L_KK) is a substitution per row (thread = row); Z_RK
// = -Z_RR Y takes lane = row, Z's columns read side by side and Y's rows
// broadcast, the sum over R split over the warps that the rows leave; Z_KK
// takes a warp per entry.  (A CTA per front straight on global memory, a
// column of the gather at a time, took 3.77 ms on a 32^3 grid; now 1.77, 1.5 of
// it in the fronts of more than 32 rows, the pieces beside each other.)
// Z: MB columns of MB + 1; Y: rows of kSelYS; P: partial sums, `slices` of them
// where the rows leave warps (1: none); SM: L_KK and inv(L_KK), 8 x 8 in rows
// of 9.
constexpr int kSelNB = 8;
constexpr int kSelYS = kSelNB + 2;  // 16-byte rows, fewer conflicts than 8
constexpr int kSelLD = 9;
constexpr int kSelSm = 2 * kSelNB * kSelLD;

template <typename Sync>
__device__ __forceinline__ void sel_small_front(int s, double* Z, int LD, double* Y, double* P,
                                                int max_slices, double* SM, int warp, int nw,
                                                Sync&& sync, const FrontDesc* __restrict__ fronts,
                                                const int* __restrict__ relmap,
                                                const double* __restrict__ Ls,
                                                double* __restrict__ Zs, double* __restrict__ Zu,
                                                const int64_t* __restrict__ zuoff) {
    constexpr int NB = kSelNB;
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, tid = 32 * warp + lane;
    const FrontDesc f = fronts[s];
    const int m = f.m, c = f.c, u = m - c;
    double *Lk = SM, *Wk = SM + NB * kSelLD;
    // this thread's row of the block's columns of L, and its entry of L_KK
    double l[NB], lk = 0.0;
    auto load = [&](int k0) {
        const int k1 = min(k0 + NB, c), r = k1 + tid;
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            l[k] = 0.0;
            if (k0 + k < c && r < m) l[k] = Ls[f.loff + r + (int64_t)(k0 + k) * f.ldl];
        }
    };
    auto load_diag = [&](int k0) {
        for (int e = tid; e < NB * NB; e += 32 * nw) {
            const int i = e & (NB - 1), j = e / NB;
            lk = 0.0;
            if (k0 + i < c && i >= j) lk = Ls[f.loff + k0 + i + (int64_t)(k0 + j) * f.ldl];
            Lk[i * kSelLD + j] = lk;
        }
    };
    load((c - 1) & ~(NB - 1));
    // the update part: the parent's Z on this front's update rows
    if (f.parent >= 0 && u > 0) {
        const FrontDesc p = fronts[f.parent];
        const int64_t zp = zuoff[f.parent], zf = zuoff[s];
        const int* rm = relmap + f.rows_off + c;
        for (int j0 = NB * warp; j0 < u; j0 += NB * nw) {
            const int rj = j0 + (lane & 7) < u ? rm[j0 + (lane & 7)] : 0;
            for (int i0 = j0 & ~31; i0 < u; i0 += 32) {
                const int i = i0 + lane;
                const int ri = i < u ? rm[i] : 0;
                double v[NB];
#pragma unroll
                for (int e = 0; e < NB; ++e) {
                    const int col = __shfl_sync(ALL, rj, e);
                    v[e] = 0.0;
                    if (i < u && i >= j0 + e) v[e] = zelem(Zs, Zu, p, zp, ri, col);
                }
#pragma unroll
                for (int e = 0; e < NB; ++e) {
                    const int j = j0 + e;
                    if (i >= u || i < j) continue;
                    Z[(c + i) + (c + j) * LD] = Z[(c + j) + (c + i) * LD] = v[e];
                    Zu[zf + i + (int64_t)j * f.ldu] = v[e];
                }
            }
        }
    }
    for (int k0 = (c - 1) & ~(NB - 1); k0 >= 0; k0 -= NB) {
        const int k1 = min(k0 + NB, c), nb = k1 - k0, nR = m - k1;
        load_diag(k0);
        sync();
        // Y = L_RK inv(L_KK), from the last column; padding columns stay zero
        if (tid < nR) {
            double y[NB];
#pragma unroll
            for (int j = NB - 1; j >= 0; --j) {
                double v = l[j];
#pragma unroll
                for (int k = j + 1; k < NB; ++k) v -= y[k] * Lk[k * kSelLD + j];
                y[j] = j < nb ? v / Lk[j * kSelLD + j] : 0.0;
            }
#pragma unroll
            for (int j = 0; j < NB; ++j) Y[tid * kSelYS + j] = y[j];
        }
        if (k0 >= NB) load(k0 - NB);
        // W = inv(L_KK), a column per lane of the last warp
        if (warp == nw - 1 && lane < nb) {
            double w[NB];
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                double v = i == lane ? 1.0 : 0.0;
#pragma unroll
                for (int k = 0; k < i; ++k) v -= Lk[i * kSelLD + k] * w[k];
                w[i] = i < nb && i >= lane ? v / Lk[i * kSelLD + i] : 0.0;
                Wk[i * kSelLD + lane] = w[i];
            }
        }
        sync();
        // Z_RK = -Z_RR Y
        const int RB = (nR + 31) / 32, NS = RB > 0 ? max(1, min(max_slices, nw / RB)) : 1;
        const int per = (nR + NS - 1) / NS;
        auto put = [&](int a, const double (&v)[NB]) {
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                if (j >= nb) continue;
                Z[(k1 + a) + (k0 + j) * LD] = Z[(k0 + j) + (k1 + a) * LD] = -v[j];
                Zs[f.loff + k1 + a + (int64_t)(k0 + j) * f.ldl] = -v[j];
            }
        };
        for (int t = warp; t < RB * NS; t += nw) {
            const int rb = t % RB, sl = t / RB, a = 32 * rb + lane;
            double acc[NB];
#pragma unroll
            for (int j = 0; j < NB; ++j) acc[j] = 0.0;
            const int b1 = min(nR, (sl + 1) * per);
#pragma unroll 2
            for (int b = sl * per; b < b1; ++b) {
                const double z = a < nR ? Z[(k1 + a) + (k1 + b) * LD] : 0.0;
                const double2* y = reinterpret_cast<const double2*>(Y + b * kSelYS);
#pragma unroll
                for (int j = 0; j < NB / 2; ++j) {
                    const double2 yy = y[j];
                    acc[2 * j] += z * yy.x;
                    acc[2 * j + 1] += z * yy.y;
                }
            }
            if (NS == 1) {
                if (a < nR) put(a, acc);
            } else {
                double2* o = reinterpret_cast<double2*>(P + (int64_t)(t * 32 + lane) * kSelYS);
#pragma unroll
                for (int j = 0; j < NB / 2; ++j) o[j] = make_double2(acc[2 * j], acc[2 * j + 1]);
            }
        }
        sync();
        if (NS > 1) {  // the slices in order
            if (tid < nR) {
                double acc[NB];
#pragma unroll
                for (int j = 0; j < NB; ++j) acc[j] = 0.0;
                for (int sl = 0; sl < NS; ++sl)
#pragma unroll
                    for (int j = 0; j < NB; ++j) acc[j] += P[(sl * RB * 32 + tid) * kSelYS + j];
                put(tid, acc);
            }
            sync();
        }
        // Z_KK = W'W - Y' Z_RK, lower part, a warp per entry
        for (int e = warp; e < nb * nb; e += nw) {
            const int i = e % nb, j = e / nb;
            if (i < j) continue;
            double v = 0.0;
            for (int a = lane; a < nR; a += 32) v -= Y[a * kSelYS + i] * Z[(k1 + a) + (k0 + j) * LD];
            if (lane >= i && lane < nb) v += Wk[lane * kSelLD + i] * Wk[lane * kSelLD + j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(ALL, v, o);
            if (lane == 0) {
                Z[(k0 + i) + (k0 + j) * LD] = Z[(k0 + j) + (k0 + i) * LD] = v;
                Zs[f.loff + k0 + i + (int64_t)(k0 + j) * f.ldl] = v;
            }
        }
        sync();
    }
}

// shared memory (doubles) of a front of up to MB rows with nw warps
__host__ __device__ constexpr int sel_slices(int MB, int nw) {
    return nw == 1 || MB > 128 ? 1 : nw;
}
__host__ __device__ constexpr size_t sel_small_doubles(int MB, int nw) {
    return (((size_t)MB * (MB + 1) + 1) & ~(size_t)1) + (size_t)MB * kSelYS +
           (sel_slices(MB, nw) > 1 ? (size_t)nw * 32 * kSelYS : 0) + kSelSm;
}

// Fronts of up to MB rows, more than 32: a CTA of eight warps each (every
// row a thread); up to 32: a warp each.
constexpr int kSelTinyRows = 32;
template <bool TINY>
__global__ void __launch_bounds__(256)
    k_selinv_front(const FrontDesc* __restrict__ fronts, const int* __restrict__ list, int nlist,
                   int MB, const int* __restrict__ relmap, const double* __restrict__ Ls,
                   double* __restrict__ Zs, double* __restrict__ Zu,
                   const int64_t* __restrict__ zuoff) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, nw = TINY ? 1 : blockDim.x >> 5;
    const int MR = TINY ? kSelTinyRows : MB, LD = MR + 1;
    double* Z = reinterpret_cast<double*>(smem_raw) +
                (TINY ? warp * sel_small_doubles(kSelTinyRows, 1) : 0);
    double* Y = Z + ((MR * LD + 1) & ~1);
    double* P = Y + MR * kSelYS;
    const int slices = sel_slices(MR, nw);
    double* SM = P + (slices > 1 ? nw * 32 * kSelYS : 0);
    if (TINY) {
        const int k = blockIdx.x * (blockDim.x >> 5) + warp;
        if (k < nlist)
            sel_small_front(list[k], Z, LD, Y, P, slices, SM, 0, 1, [] { __syncwarp(); }, fronts,
                            relmap, Ls, Zs, Zu, zuoff);
    } else {
        sel_small_front(list[blockIdx.x], Z, LD, Y, P, slices, SM, warp, nw,
                        [] { __syncthreads(); }, fronts, relmap, Ls, Zs, Zu, zuoff);
    }
}

// ---------------------------------------------------------------------------
// large fronts: the same recurrence in blocks of kSelT = 64 pivot columns
// (the factor's diagonal tiles, whose inverses W it stored), many CTAs per
// front, per level one gather of Z_UU from the parent's Z (CTA per front and
// 16 columns), then per block step over every large front of the level:
//   zrk     Z_RK = -Z_RR Y, CTA per front, 64-row tile of R and split of the
//           sum over R, as partial 64 x 64 sums; the same launch computes the
//           next step's Y = L_RK W (it needs only L)
//   fin     the partial sums added in split order, Z_RK written, and the
//           tile's part of Y' Z_RK kept for zkk (done by zrk itself where a
//           launch has tiles enough and the sum is not split)
//   zkk     Z_KK = W'W - Y' Z_RK, eight CTAs per front
// The products are FP64 matrix instructions over gathered operands
// (tile64.cuh).  A step is a chain of three launches, so the sums are split
// until the launch has three CTAs for every SM.  32^3 grid (root of 2108
// columns: 33 steps of up to 33 x 33 tiles): 5.4 ms in all, against 36.4 ms
// with one CTA per tile row, register FMAs and a front's Y' Z_RK on one CTA.
// Y of the even and the odd steps sit in the front's scratch (2 m x 64).
// ---------------------------------------------------------------------------

constexpr int kSelT = 64;
constexpr int kSelSlabs = 8;  // CTAs of zkk per front

__device__ __forceinline__ const double* zat(const double* __restrict__ Zs,
                                             const double* __restrict__ Zu, const FrontDesc& f,
                                             int64_t zoff, int r, int col) {
    if (r < col) {
        const int t = r;
        r = col;
        col = t;
    }
    return col < f.c ? Zs + f.loff + r + (int64_t)col * f.ldl
                     : Zu + zoff + (r - f.c) + (int64_t)(col - f.c) * f.ldu;
}

struct SelStep {
    int kb, k0, k1, nb;
};
__device__ __forceinline__ SelStep sel_step(const FrontDesc& f, int step) {
    SelStep t;
    const int nblk = (f.c + kSelT - 1) / kSelT;
    t.kb = nblk - 1 - step;
    t.k0 = t.kb * kSelT;
    t.k1 = min(t.k0 + kSelT, f.c);
    t.nb = t.k1 - t.k0;
    return t;
}

__global__ void __launch_bounds__(256)
    k_sel_gather(const FrontDesc* __restrict__ fronts, const int* __restrict__ items,
                 const int* __restrict__ before, int nitems, const int* __restrict__ relmap,
                 double* __restrict__ Zs, double* __restrict__ Zu,
                 const int64_t* __restrict__ zuoff) {
    const int it = find_item(before, nitems, blockIdx.x);
    const int s = items[it], blk = blockIdx.x - before[it];
    const FrontDesc f = fronts[s];
    const FrontDesc p = fronts[f.parent];
    const int u = f.m - f.c;
    const int lane = threadIdx.x & 31;
    const int64_t zf = zuoff[s], zp = zuoff[f.parent];
    const int* rm = relmap + f.rows_off + f.c;
    for (int b = 16 * blk + (threadIdx.x >> 5); b < min(16 * blk + 16, u); b += 8) {
        const int pb = rm[b];
        // the parent's column, by front row
        const double* src = pb < p.c ? Zs + p.loff + (int64_t)pb * p.ldl
                                     : Zu + zp - p.c + (int64_t)(pb - p.c) * p.ldu;
        double* dst = Zu + zf + (int64_t)b * f.ldu;
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

// a launch's work list on the device: item k of CTAs before[k] .. before[k + 1]
struct SelList {
    const int* items;
    const int* before;
    int nitems, nctas, step;
};
struct SelData {
    const FrontDesc* fronts;
    const double* Ls;
    const double* Dinv;
    const int64_t* dinv_off;
    double* Zs;
    double* Zu;
    const int64_t* zuoff;
    double* Yscr;
    const int64_t* yoff;
    double* part;  // 64 x 64 partial sums of Z_RK, then of Y' Z_RK
    double* Q;
    // Y of a step ((m - k1) x 64, row-major)
    __device__ double* Y(int s, const FrontDesc& f, int step) const {
        return Yscr + yoff[s] + (int64_t)(step & 1) * f.m * kSelT;
    }
};

// one 64-row tile of Y = L_RK W
__device__ void sel_y_tile(const SelData& D, const SelList& w, int cta, double* sm) {
    using namespace t64;
    const int it = find_item(w.before, w.nitems, cta);
    const int s = w.items[it];
    const FrontDesc f = D.fronts[s];
    const SelStep t = sel_step(f, w.step);
    const int a0 = t.k1 + T * (cta - w.before[it]), rows = min(T, f.m - a0), nb = t.nb;
    const double* L = D.Ls + f.loff + a0 + (int64_t)t.k0 * f.ldl;
    const double* W = D.Dinv + D.dinv_off[s] + (int64_t)t.kb * T * T;
    Acc acc;
    zero(acc);
    product<false, true>(
        sm, 0, nb,
        op(L, [=](int k, int x) { return k < nb && x < rows ? L + x + (int64_t)k * f.ldl : nullptr; }),
        op(W, [=](int k, int x) { return k < nb ? W + k + x * T : nullptr; }), acc);
    double* Y = D.Y(s, f, w.step) + (int64_t)(a0 - t.k1) * T;
    each(acc, [&](int r, int c, double v) {
        if (r < rows) Y[(int64_t)r * T + c] = v;
    });
}

// the finished 64 x 64 sum of Z_RR Y at rows a0 ..: Z_RK and the tile's Y' Z_RK
__device__ void sel_finish(const SelData& D, const FrontDesc& f, const SelStep& t, const double* Y,
                           int a0, int rows, const t64::Acc& acc, double* sm, double* q) {
    using namespace t64;
    double* Zt = sm;           // [row][column of the block]
    double* Yt = sm + T * LD;  // [row][column of the block]
    each(acc, [&](int r, int c, double v) {
        Zt[r * LD + c] = r < rows ? -v : 0.0;
        if (r < rows && c < t.nb) D.Zs[f.loff + a0 + r + (int64_t)(t.k0 + c) * f.ldl] = -v;
    });
    for (int e = threadIdx.x; e < T * T; e += THREADS) {
        const int r = e / T, c = e % T;
        Yt[r * LD + c] = r < rows ? Y[(int64_t)(a0 - t.k1 + r) * T + c] : 0.0;
    }
    __syncthreads();
    Acc z;
    zero(z);
    for (int k = 0; k < T; k += 16) step16(Yt + k * LD, Zt + k * LD, z);
    each(z, [&](int r, int c, double v) { q[r * T + c] = v; });
}

template <bool SPLIT>
__global__ void __launch_bounds__(t64::THREADS, 3)
    k_sel_zrk(SelData D, SelList w, int nsplit, SelList next) {
    using namespace t64;
    extern __shared__ __align__(16) double sel_sm[];
    if ((int)blockIdx.x >= w.nctas * nsplit) {
        sel_y_tile(D, next, blockIdx.x - w.nctas * nsplit, sel_sm);
        return;
    }
    const int cta = blockIdx.x / nsplit, ks = blockIdx.x % nsplit;
    const int it = find_item(w.before, w.nitems, cta);
    const int s = w.items[it];
    const FrontDesc f = D.fronts[s];
    const SelStep t = sel_step(f, w.step);
    const int a0 = t.k1 + T * (cta - w.before[it]), rows = min(T, f.m - a0);
    const int64_t zf = (f.parent >= 0 && f.m > f.c) ? D.zuoff[s] : -1;
    const double* Y = D.Y(s, f, w.step);
    // this split's tiles of R
    const int nt = (f.m - t.k1 + T - 1) / T;
    const int b0 = t.k1 + T * (int)((int64_t)ks * nt / nsplit);
    const int b1 = min(f.m, t.k1 + T * (int)((int64_t)(ks + 1) * nt / nsplit));
    Acc acc;
    zero(acc);
    auto z = op(D.Zs, [&](int k, int x) -> const double* {
        return k < b1 && x < rows ? zat(D.Zs, D.Zu, f, zf, a0 + x, k) : nullptr;
    });
    auto y = op(Y, [&](int k, int x) -> const double* {
        return k < b1 ? Y + (int64_t)(k - t.k1) * T + x : nullptr;
    });
    // columns of R before this row tile are stored along its rows, the others
    // along theirs
    const int mid = min(max(a0 + T, b0), b1);
    if (b0 < mid) {
        auto z0 = op(D.Zs, [&](int k, int x) -> const double* {
            return k < mid && x < rows ? zat(D.Zs, D.Zu, f, zf, a0 + x, k) : nullptr;
        });
        auto y0 = op(Y, [&](int k, int x) -> const double* {
            return k < mid ? Y + (int64_t)(k - t.k1) * T + x : nullptr;
        });
        product<false, false>(sel_sm, b0, mid, z0, y0, acc);
    }
    if (mid < b1) product<true, false>(sel_sm, mid, b1, z, y, acc);
    if constexpr (SPLIT) {
        double* p = D.part + (int64_t)blockIdx.x * T * T;
        each(acc, [&](int r, int c, double v) { p[r * T + c] = v; });
    } else {
        sel_finish(D, f, t, Y, a0, rows, acc, sel_sm, D.Q + (int64_t)cta * T * T);
    }
}

__global__ void __launch_bounds__(t64::THREADS, 3) k_sel_fin(SelData D, SelList w, int nsplit) {
    using namespace t64;
    extern __shared__ __align__(16) double sel_sm[];
    const int cta = blockIdx.x;
    const int it = find_item(w.before, w.nitems, cta);
    const int s = w.items[it];
    const FrontDesc f = D.fronts[s];
    const SelStep t = sel_step(f, w.step);
    const int a0 = t.k1 + T * (cta - w.before[it]), rows = min(T, f.m - a0);
    Acc acc;
    zero(acc);
    for (int ks = 0; ks < nsplit; ++ks) {
        const double* p = D.part + ((int64_t)cta * nsplit + ks) * T * T;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
        const int wr = (warp & 1) * 32, wc = (warp >> 1) * 32;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const double* e = p + (wr + 16 * m + 2 * g + r) * T + wc + 16 * n + 4 * q;
                    const double2 u = *reinterpret_cast<const double2*>(e);
                    const double2 v = *reinterpret_cast<const double2*>(e + 2);
                    acc[m][n][0][2 * r] += u.x;
                    acc[m][n][1][2 * r] += u.y;
                    acc[m][n][0][2 * r + 1] += v.x;
                    acc[m][n][1][2 * r + 1] += v.y;
                }
    }
    sel_finish(D, f, t, D.Y(s, f, w.step), a0, rows, acc, sel_sm, D.Q + (int64_t)cta * T * T);
}

__global__ void __launch_bounds__(256) k_sel_zkk(SelData D, SelList w) {
    constexpr int T = kSelT;
    __shared__ double Ws[T * (T + 1)];
    const int it = blockIdx.x / kSelSlabs, slab = blockIdx.x % kSelSlabs;
    const int s = w.items[it];
    const FrontDesc f = D.fronts[s];
    const SelStep t = sel_step(f, w.step);
    if (slab * (T / kSelSlabs) >= t.nb) return;
    const double* W = D.Dinv + D.dinv_off[s] + (int64_t)t.kb * T * T;
    for (int e = threadIdx.x; e < T * T; e += 256) Ws[(e & 63) * (T + 1) + (e >> 6)] = W[e];
    __syncthreads();
    const int cta0 = w.before[it], cta1 = w.before[it + 1];
    for (int e = threadIdx.x; e < T * (T / kSelSlabs); e += 256) {
        const int j = slab * (T / kSelSlabs) + e % (T / kSelSlabs), i = e / (T / kSelSlabs);
        if (i < j || i >= t.nb) continue;
        double neg = 0.0, pos = 0.0;
        const double* q = D.Q + (int64_t)cta0 * T * T + i * T + j;
#pragma unroll 8
        for (int b = cta0; b < cta1; ++b, q += T * T) neg += *q;
        for (int k = i; k < t.nb; ++k) pos += Ws[k * (T + 1) + i] * Ws[k * (T + 1) + j];
        D.Zs[f.loff + (t.k0 + i) + (int64_t)(t.k0 + j) * f.ldl] = pos - neg;
    }
}

// G (caller order; zeroed by the caller) of every lower-triangle entry e:
// its front position (a_pos: row | column << 16 within front a_front[e]).
__global__ void k_grad_lower(int nnz, const FrontDesc* __restrict__ fronts,
                             const int* __restrict__ a_front, const int* __restrict__ a_src,
                             const int* __restrict__ a_pos, const int* __restrict__ rows,
                             const int* __restrict__ perm, const double* __restrict__ Zs,
                             const double* __restrict__ x, double* __restrict__ G) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += gridDim.x * blockDim.x) {
        const int src = a_src[e];
        if (src < 0) continue;  // a duplicate the assembly drops: gradient 0
        const FrontDesc f = fronts[a_front[e]];
        const int pos = a_pos[e], r = pos & 0xffff, jj = pos >> 16;
        double z = Zs[f.loff + r + (int64_t)jj * f.ldl];
        const int pr = rows[f.rows_off + r], pc = f.first_col + jj;
        if (x) {
            const int i = perm ? perm[pr] : pr, j = perm ? perm[pc] : pc;
            z -= x[i] * x[j];
        }
        G[src] = pr == pc ? z : 2.0 * z;
    }
}

// logdet = 2 sum log L(j, j): per block a fixed-order sum over its
// supernodes, a lane each, the wider ones then a warp each (a root of thousands of
// columns read by one thread took 1.1 ms, a warp for every column of a 300 x 300
// grid's nodal tree 20 us more than a lane), then one block sums the partials
// (deterministic)
template <typename T>
__global__ void k_logdet_partial(int nsuper, const FrontDesc* __restrict__ fronts,
                                 const T* __restrict__ Ls, double* __restrict__ partial) {
    __shared__ double red[256];
    double v = 0.0;
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5, nw = gridDim.x * wpb;
    for (int s0 = blockIdx.x * wpb + (threadIdx.x >> 5); s0 < nsuper; s0 += 32 * nw) {
        const int s = s0 + lane * nw;  // neighbours in the tree to different warps
        int c = 0;
        int64_t off = 0, step = 0;
        if (s < nsuper) {
            const FrontDesc& f = fronts[s];
            c = f.c, off = f.loff, step = f.ldl + 1;
        }
        if (c <= 4)
            for (int j = 0; j < c; ++j) v += log((double)Ls[off + j * step]);
        for (unsigned wide = __ballot_sync(0xffffffffu, c > 4); wide; wide &= wide - 1) {
            const int h = __ffs(wide) - 1, hc = __shfl_sync(0xffffffffu, c, h);
            const int64_t hoff = __shfl_sync(0xffffffffu, off, h);
            const int64_t hstep = __shfl_sync(0xffffffffu, step, h);
            for (int j = lane; j < hc; j += 32) v += log((double)Ls[hoff + j * hstep]);
        }
    }
    red[threadIdx.x] = v;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

__global__ void k_logdet_final(int nparts, const double* __restrict__ partial,
                               double* __restrict__ out) {
    __shared__ double red[256];
    double v = 0.0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) v += partial[i];
    red[threadIdx.x] = v;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = 2.0 * red[0];
}

constexpr int kLogdetBlocks = 148 * 2;

// splits of a step's sums: until the launch has three CTAs per SM
static int sel_splits(int nctas, int num_sms) {
    const int want = 3 * num_sms;
    return nctas >= want || nctas == 0 ? 1 : std::min((want + nctas - 1) / nctas, 16);
}
// doubles of the partial sums and of the Y' Z_RK parts over every step
int64_t selinv_partials(const DevPlan& D) {
    int64_t p = 1, q = 1;
    for (const WorkList& w : D.sel.h_steps) {
        const int ns = sel_splits(w.nctas, D.num_sms);
        if (ns > 1) p = std::max<int64_t>(p, (int64_t)w.nctas * ns);
        q = std::max<int64_t>(q, w.nctas);
    }
    return (p + q) * kSelT * kSelT;
}

// Level by level from the root: the small fronts (k_selinv_front) in pieces on
// streams of their own, the large fronts by the tiled
// phases above beside them, block step by block step (fronts with fewer
// pivot blocks join the later steps).
void launch_selinv(const DevPlan& D, const double* Ls, const double* Dinv, double* Zs,
                   double* Zu, double* Yscr, double* part, cudaStream_t st) {
    const SelSchedule& S = D.sel;
    int64_t psize = 1;
    for (const WorkList& w : S.h_steps) {
        const int ns = sel_splits(w.nctas, D.num_sms);
        if (ns > 1) psize = std::max<int64_t>(psize, (int64_t)w.nctas * ns);
    }
    const SelData data{D.fronts, Ls, Dinv, D.dinv_off, Zs, Zu, D.zuoff, Yscr, D.yoff,
                       part, part + psize * kSelT * kSelT};
    auto list = [&](const WorkList& w) {
        return SelList{S.items + w.off, S.before + w.off, w.nitems, w.nctas, w.step};
    };
    const SelList none{nullptr, nullptr, 0, 0, 0};
    constexpr size_t SM = t64::SMEM_BYTES;
    for (int l = D.nlevels - 1; l >= 0; --l) {
        const int sb = D.h_small_ptr[l * kSmallBuckets], se = D.h_small_ptr[(l + 1) * kSmallBuckets];
        const int q0 = S.h_step_beg[l], q1 = S.h_step_beg[l + 1];
        // the pieces of the small fronts: at most 32 rows, then each size bucket
        int pb[DevPlan::kSmallPieces + 1], npieces = 0;
        pb[0] = sb;
        for (int i = 0; i < DevPlan::kSmallPieces; ++i) {
            pb[i + 1] = D.h_small_ptr[l * kSmallBuckets + Plan::kTinyBuckets + i];
            npieces += pb[i + 1] > pb[i];
        }
        const bool fork = D.piece_st[0] && npieces > 0 && npieces + (q1 > q0) > 1;
        if (fork) cudaEventRecord(D.fork_ev, st);
        for (int i = 0; i < DevPlan::kSmallPieces; ++i) {
            const int n = pb[i + 1] - pb[i];
            if (n == 0) continue;
            const cudaStream_t ss = fork ? D.piece_st[i] : st;
            if (fork) cudaStreamWaitEvent(ss, D.fork_ev, 0);
            if (i == 0) {
                k_selinv_front<true><<<(n + 7) / 8, 256,
                                       8 * sel_small_doubles(kSelTinyRows, 1) * sizeof(double),
                                       ss>>>(D.fronts, D.small_list + pb[i], n, kSelTinyRows,
                                             D.relmap, Ls, Zs, Zu, D.zuoff);
            } else {
                const int MB = Plan::small_limit[Plan::kTinyBuckets + i - 1];
                k_selinv_front<false><<<n, 256, sel_small_doubles(MB, 8) * sizeof(double), ss>>>(
                    D.fronts, D.small_list + pb[i], n, MB, D.relmap, Ls, Zs, Zu, D.zuoff);
            }
            if (fork) cudaEventRecord(D.piece_join[i], ss);
        }
        if (q1 > q0) {
            const SelList y = list(S.h_steps[q0]);
            if (y.nctas > 0)
                k_sel_zrk<false><<<y.nctas, t64::THREADS, SM, st>>>(data, none, 1, y);
        }
        const WorkList& g = S.h_gather[l];
        if (g.nctas > 0)
            k_sel_gather<<<g.nctas, 256, 0, st>>>(D.fronts, S.items + g.off, S.before + g.off,
                                                  g.nitems, D.relmap, Zs, Zu, D.zuoff);
        for (int q = q0; q < q1; ++q) {
            const SelList w = list(S.h_steps[q]);
            const SelList next = q + 1 < q1 ? list(S.h_steps[q + 1]) : none;
            const int ns = sel_splits(w.nctas, D.num_sms);
            const int grid = w.nctas * ns + next.nctas;
            if (ns > 1) {
                k_sel_zrk<true><<<grid, t64::THREADS, SM, st>>>(data, w, ns, next);
                k_sel_fin<<<w.nctas, t64::THREADS, SM, st>>>(data, w, ns);
            } else if (grid > 0) {
                k_sel_zrk<false><<<grid, t64::THREADS, SM, st>>>(data, w, ns, next);
            }
            k_sel_zkk<<<w.nitems * kSelSlabs, 256, 0, st>>>(data, w);
        }
        for (int i = 0; i < DevPlan::kSmallPieces; ++i)
            if (fork && pb[i + 1] > pb[i]) cudaStreamWaitEvent(st, D.piece_join[i], 0);
    }
}

void launch_grad_lower(const DevPlan& D, int nnz, const int* perm, const double* Zs,
                       const double* x, double* G, cudaStream_t st) {
    const int blocks = std::max(1, std::min((nnz + 255) / 256, 148 * 8));
    k_grad_lower<<<blocks, 256, 0, st>>>(nnz, D.fronts, D.a_front, D.a_src, D.a_pos, D.rows, perm,
                                         Zs, x, G);
}

template <typename T>
void launch_logdet(const DevPlan& D, const T* Ls, double* partial, double* out, cudaStream_t st) {
    k_logdet_partial<T><<<kLogdetBlocks, 256, 0, st>>>(D.nsuper, D.fronts, Ls, partial);
    k_logdet_final<<<1, 256, 0, st>>>(kLogdetBlocks, partial, out);
}
template void launch_logdet<double>(const DevPlan&, const double*, double*, double*, cudaStream_t);
template void launch_logdet<float>(const DevPlan&, const float*, double*, double*, cudaStream_t);

int logdet_partials() { return kLogdetBlocks; }

void init_selinv() {
    const int sm = (int)t64::SMEM_BYTES;
    cudaFuncSetAttribute(k_sel_zrk<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_sel_zrk<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_selinv_front<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         227 * 1024);
    cudaFuncSetAttribute(k_selinv_front<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         227 * 1024);
    cudaFuncSetAttribute(k_sel_fin, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
}
int selinv_tile() { return kSelT; }

}  // namespace mdgpu
