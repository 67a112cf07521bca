// Supernodal triangular solves L y = b (forward, leaves to root) and
// L' x = y (backward, root to leaves) on the panel storage of the factor.
//
// Forward is multifrontal like the factor: supernode s forms its front vector
// f (m_s x nrhs) from the right-hand side rows of its pivot columns and the
// update parts of its children's front vectors (pulled child by child, so the
// sums are deterministic), solves with the diagonal block, and leaves
// f[c:m] - L21 y as its own update part.  Backward reads the already final
// solution entries of its update rows (ancestors) directly.
//
// Small fronts: a warp (or a part of one) per front.  Large fronts: tasks of
// 64-row tiles; a pivot tile applies its block's inverse (stored by the
// factorization), a 64 x 64 product instead of a serial substitution.
#include <algorithm>
#include <type_traits>

#include "device_common.cuh"
#include "kernels.hpp"

namespace mdgpu {

// Front vector of supernode s: rows fv_off[s] .. fv_off[s] + m - 1 of one
// array whose row holds the nrhs right-hand sides side by side, so row r,
// right-hand side q is front_vec(...)[r * nrhs + q].
__device__ inline double* front_vec(double* fv, const int64_t* fv_off, int s, int nrhs) {
    return fv + fv_off[s] * nrhs;
}

// ---------------------------------------------------------------------------
// one launch per direction: dependency-ordered work items
//
// Each CTA takes the next item by an atomic ticket, so every item that
// started before it holds a lower ticket; the lists are ordered so that an
// item only waits for items earlier in its list, hence for CTAs that are
// already resident, and the waits cannot deadlock.  A consumer polls the values
// themselves with an iteration limit, after which the solve is aborted (every
// waiter leaves) and the error word is set for the host.
// ---------------------------------------------------------------------------

constexpr int kSolveWaitPolls = 1 << 18;  // ~0.1-0.3 s at ~1 us per poll
constexpr int kVecLD = kTile + 4;  // column stride of a vector block in shared memory: 4 mod 16
                                   // doubles, a conflict-free operand of the matrix instructions
constexpr int kGroupRhs = 8;       // right-hand sides of one group (a matrix instruction's columns)

__device__ __forceinline__ int ld_relaxed_gpu(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// Published values.  Everything that one task of a launch hands to another
// -- a front's update rows, a pivot tile's solution, the backward partial sums,
// the solution rows -- sits in words preset to the all-ones bit pattern (a NaN
// that arithmetic never produces), and a producer stores final values only
// (aligned 8-byte stores are single-copy atomic), so a consumer that sees no
// sentinel has the data: one trip through L2 hands a value over, where a
// fence, a counter and a poll of it took three.  A chain of one-column fronts of
// 5 rows, FP64: 0.7 + 1.0 us per front forward and backward (4.8 + 4.1 with
// counters); 24 x 23 grid 203 + 159 us -> 32 + 32; 333 x 257 grid FP32, three
// right-hand sides 0.97 + 0.85 ms -> 0.35 + 0.44.
__device__ __forceinline__ double ld_relaxed_f64(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
// every publication goes through here: a NaN that carries the sentinel's
// all-ones pattern (a right-hand side's own payload passed along) is
// published as the default NaN, so a slot is never read as unpublished once
// written
__device__ __forceinline__ void st_relaxed_f64(double* p, double v) {
    if (__double_as_longlong(v) == -1ll) v = __longlong_as_double(0x7ff8000000000000ll);
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ bool is_unpublished(double v) {
    return __double_as_longlong(v) == -1ll;
}
struct SolveAbort {
    int* flag;
    int* err;
};

// All threads of the CTA poll a slot together (uniform result): the warps that
// hold slot elements spin on their own elements (a warp vote per round, no
// block barrier, a short sleep and an abort check every 32 rounds), the others
// go straight to the closing barrier; with an iteration limit, after which the
// launch is aborted and the error word set.
// (src: the slot, column after column of 64 rows; dst: columns kVecLD apart)
__device__ bool poll_published(double* dst, const double* src, int nk, int nrhs,
                               const SolveAbort& ab) {
    constexpr int T = kTile;
    const int total = T * nrhs, lane = threadIdx.x & 31;  // total: a multiple of 64
    bool ok = true;
    for (int base = threadIdx.x & ~31; ok && base < total; base += blockDim.x) {
        const int e = base + lane;
        const bool need = (e & (T - 1)) < nk;
        double v = 0.0;
        for (int it = 0;; ++it) {
            if (need) v = ld_relaxed_f64(src + e);
            if (__all_sync(0xffffffffu, !need || !is_unpublished(v))) break;
            if (it + 1 >= kSolveWaitPolls) {
                if (lane == 0) {
                    atomicExch(ab.flag, 1);
                    atomicOr(ab.err, 1);
                }
                ok = false;
                break;
            }
            if ((it & 31) == 31) {
                const int a = lane == 0 ? ld_relaxed_gpu(ab.flag) : 0;
                if (__shfl_sync(0xffffffffu, a, 0)) {
                    ok = false;
                    break;
                }
                __nanosleep(32);
            }
        }
        if (ok) dst[(e / T) * kVecLD + (e & (T - 1))] = need ? v : 0.0;
    }
    return __syncthreads_and(ok);
}

// NQ neighbouring published values p[0 .. nq - 1]: a first look (the loads of
// several places are issued together).
template <int NQ>
__device__ __forceinline__ void peek_values(const double* p, bool need, int nq, double (&v)[NQ]) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        v[q] = 0.0;
        if (need && q < nq) v[q] = ld_relaxed_f64(p + q);
    }
}

// Then the wait for the ones not there yet, with a short sleep between the
// looks, by the lanes of `mask` together (converged), each with values from
// R places: the rounds are uniform, so the lanes leave converged.  After loops
// of their own lanes ran the rest of a front in pieces, also past a
// __syncwarp, and every shuffle waited about 500 cycles for the pieces to meet
// (8 us per front in the chain above).  at(k): place k, which a lane needs
// where v[k] is unpublished.
template <int R, int NQ, typename F>
__device__ __forceinline__ void await_together(F&& at, int nq, double (&v)[R][NQ], unsigned mask,
                                               const SolveAbort& ab) {
    for (int it = 1;; ++it) {
        bool miss = false;
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
            for (int q = 0; q < NQ; ++q) miss = miss || is_unpublished(v[k][q]);
        if (!__any_sync(mask, miss)) return;
        if (it > 2) __nanosleep(it < 64 ? 40 : 200);
        if ((it & 15) == 0) {
            if (miss && it >= kSolveWaitPolls) {
                atomicExch(ab.flag, 1);
                atomicOr(ab.err, 1);
            }
            if (__any_sync(mask, ld_relaxed_gpu(ab.flag))) return;
        }
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (is_unpublished(v[k][q])) v[k][q] = ld_relaxed_f64(at(k) + q);
    }
}

// four neighbouring elements on 16 bytes
__device__ __forceinline__ void ld4(const float* p, float (&v)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&v)[4]) {
    const double2 a = *reinterpret_cast<const double2*>(p);
    const double2 b = *reinterpret_cast<const double2*>(p + 2);
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
}

// Backward, update-row gathers: the solution rows of a front's ancestors are
// final once its parent's first pivot row (at global column pcol; none for a
// root) is: a large front publishes its tiles from the last, and the rows above
// the parent came before it.  One warp waits for that row, as many gathers wait
// for the same few.
__device__ __forceinline__ void await_parent(int pcol, const double* xs, int nrhs,
                                             const SolveAbort& ab) {
    if (pcol < 0) return;
    const double* p = xs + (int64_t)pcol * nrhs;
    double v[1][1] = {{ld_relaxed_f64(p)}};
    await_together<1, 1>([&](int) { return p; }, 1, v, 0xffffffffu, ab);
}

__device__ __forceinline__ void cp_async_commit_group() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait_groups() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Stage layout of a 64 x 64 block of L (or of a diagonal inverse): column-
// major, columns of blk_ld elements (a multiple of 16 bytes), copied in
// 16-byte chunks from the 16-byte boundary at or below the block's first
// row, so row r of column c sits at c * blk_ld + d + r with d =
// blk_off(first row).  Rows past the block and columns past nc are
// zero-filled by the copies themselves (source size below 16 bytes).  The L
// store's columns start on 32-byte boundaries (ldl a multiple of 8, front
// offsets of 32), the inverses' on 64 * 64 elements.
template <typename TL>
__host__ __device__ constexpr int blk_ld() {
    return kTile + 4;
}
template <typename TL>
__device__ __forceinline__ int blk_off(int start) {
    return start & (16 / (int)sizeof(TL) - 1);
}
// (blk_ld = 68: 4 mod 16 doubles and 4 mod 32 floats, the bank spread of the
// four columns that a matrix-instruction operand takes at once)
// rows start .. start + nr - 1 and columns 0 .. nc - 1 of the matrix at src
// (column stride ld)
template <typename TL>
__device__ __forceinline__ void load_block_async(TL* dst, const TL* src, int64_t ld, int start,
                                                 int nr, int nc) {
    constexpr int E = 16 / (int)sizeof(TL), LDB = blk_ld<TL>(), CH = LDB / E;
    const int r0 = start - blk_off<TL>(start);
    for (int e = threadIdx.x; e < kTile * CH; e += blockDim.x) {
        const int col = e / CH, u = e - col * CH;
        const int row = r0 + u * E;
        const int bytes = col < nc ? min(max(start + nr - row, 0), E) * (int)sizeof(TL) : 0;
        const TL* sp = bytes ? src + row + (int64_t)col * ld : src;
        const uint32_t da = static_cast<uint32_t>(__cvta_generic_to_shared(dst + col * LDB + u * E));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(da), "l"(sp), "r"(bytes)
                     : "memory");
    }
}

// ---------------------------------------------------------------------------
// large-front tile tasks: a pipeline of two or three stages streams the L blocks a
// task multiplies, each with the vector block it is multiplied by (a pivot
// tile's published solution, or gathered solution rows), by cp.async; the
// block in use is consumed while the next ones load.  Published vectors come
// through L2 (16-byte cp.async.cg); a stage whose copy still holds a
// sentinel falls back to polling that slot.
// ---------------------------------------------------------------------------

// three where they leave three CTAs per SM: one right-hand side, FP32 (two: 3.66 +
// 3.26 ms in twelve solves of the 24^3 three-unknown grid, three: 3.51 + 3.23)
template <typename TL, bool MULTI>
__host__ __device__ constexpr int solve_stages() {
    return sizeof(TL) == 4 && !MULTI ? 3 : 2;
}

// shared memory of a tile task: the stages' L blocks, their vector blocks, a
// vector, the gather's row indices; one right-hand side also keeps the
// diagonal inverse in a block of its own (several take it through the stages,
// after the last L block)
template <typename TL, bool MULTI>
__host__ __device__ constexpr size_t level_smem_bytes() {
    return ((size_t)(solve_stages<TL, MULTI>() + (MULTI ? 0 : 1)) * kTile * blk_ld<TL>()) *
               sizeof(TL) +
           (size_t)(solve_stages<TL, MULTI>() + 1) * kVecLD * (MULTI ? kGroupRhs : 1) * sizeof(double) +
           (size_t)SolveScheduleHost::kGatherTiles * kTile * sizeof(int);
}

template <typename TL, bool MULTI>
struct LevelSmem {
    static constexpr int S = solve_stages<TL, MULTI>();
    static constexpr int VB = kVecLD * (MULTI ? kGroupRhs : 1);
    TL* Lst;      // stages x T x LD
    TL* Dk;       // T x LD (one right-hand side)
    double* Vst;  // stages x VB
    double* Y;    // VB
    int* idx;     // kGatherTiles x T
    __device__ LevelSmem() {
        constexpr int T = kTile, LD = blk_ld<TL>();
        extern __shared__ __align__(16) unsigned char smem_raw[];
        Lst = reinterpret_cast<TL*>(smem_raw);
        Dk = Lst + S * T * LD;
        Vst = reinterpret_cast<double*>(Dk + (MULTI ? 0 : T * LD));
        Y = Vst + S * VB;
        idx = reinterpret_cast<int*>(Y + VB);
    }
    __device__ TL* lb(int p) const { return Lst + (p % S) * kTile * blk_ld<TL>(); }
    __device__ double* vb(int p) const { return Vst + (p % S) * VB; }
};

// a published T x nrhs slot into a stage (16-byte copies through L2; T * nrhs
// is even and slots start on 16 bytes)
__device__ __forceinline__ void load_slot_async(double* dst, const double* src, int nrhs) {
    for (int q = threadIdx.x; q < kTile * nrhs / 2; q += blockDim.x) {
        const uint32_t da = static_cast<uint32_t>(__cvta_generic_to_shared(
            dst + (2 * q / kTile) * kVecLD + ((2 * q) & (kTile - 1))));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(da), "l"(src + 2 * q)
                     : "memory");
    }
}

// After the stage's copy landed: rows >= nk zeroed, rows < nk checked for
// the sentinel; an unpublished row sends the CTA to poll the slot.  Uniform
// result; false = the solve was aborted.
__device__ __forceinline__ bool settle_slot(double* v, const double* src, int nk, int nrhs,
                                            const SolveAbort& ab) {
    bool mine = true;
    for (int e = threadIdx.x; e < kTile * nrhs; e += blockDim.x) {
        double& x = v[(e / kTile) * kVecLD + (e & (kTile - 1))];
        if ((e & (kTile - 1)) >= nk)
            x = 0.0;
        else if (is_unpublished(x))
            mine = false;
    }
    if (__syncthreads_and(mine)) return true;
    return poll_published(v, src, nk, nrhs, ab);
}

// Forward, one right-hand side, 64 x 64 blocks: thread (row r, phase g) sums
// over the column pairs 8 u + 2 g, + 1: no bank conflicts between the phases,
// the vector in 16-byte reads, four chains of sums (an FP64 multiply-add takes
// about 40 cycles to the next one that needs it, so one chain of 16 took 640
// of a tile's 3400 cycles, twice; 1.90 -> 1.75 us per tile of a chain, FP64).
// The backward sweep's column-wise reads conflict that way, and it keeps one
// chain.  B: the thread's row.
template <typename TL>
__device__ __forceinline__ double row_dot(const TL* B, const double* V, int g) {
    constexpr int LD = blk_ld<TL>();
    double a[4] = {};
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const double2 v = *reinterpret_cast<const double2*>(V + 8 * u + 2 * g);
        a[u & 3] += (double)B[(8 * u + 2 * g) * LD] * v.x;
        a[u & 3] += (double)B[(8 * u + 2 * g + 1) * LD] * v.y;
    }
    return (a[0] + a[1]) + (a[2] + a[3]);
}

// x[q] += the front-vector rows that the assembly map adds into a row (fv row
// e at fv + e * nrhs; NQ neighbouring right-hand sides), in child order, every
// entry waited for; a whole warp together, lanes with need (ar: the row's entry
// range) and without.  Most rows have at most two entries, in flight together; in
// a warp with more, eight (four of two right-hand sides) per trip: a root of 300
// rows over 2000 leaves, one right-hand side FP32, 0.39 ms, two per trip 0.62 (a
// loop of two per trip behind one of eight cost chains of large fronts 2 %).
template <int E, int NQ>
__device__ __forceinline__ void gather_some(int e, int e1, const int* __restrict__ amap_ent,
                                            const double* fv, int nrhs, int nq, double (&x)[NQ],
                                            const SolveAbort& ab) {
    const double* p[E];
    double v[E][NQ];
#pragma unroll
    for (int i = 0; i < E; ++i) {
        p[i] = fv;
        if (e + i < e1) p[i] += (int64_t)amap_ent[e + i] * nrhs;
    }
#pragma unroll
    for (int i = 0; i < E; ++i) peek_values<NQ>(p[i], e + i < e1, nq, v[i]);
    await_together<E, NQ>([&](int i) { return p[i]; }, nq, v, 0xffffffffu, ab);
#pragma unroll
    for (int i = 0; i < E; ++i)
#pragma unroll
        for (int q = 0; q < NQ; ++q) x[q] += v[i][q];
}
template <int NQ>
__device__ __forceinline__ void gather_entries(bool need, const int* ar,
                                               const int* __restrict__ amap_ent, const double* fv,
                                               int nrhs, int nq, double (&x)[NQ],
                                               const SolveAbort& ab) {
    constexpr int WIDE = NQ == 1 ? 8 : 4;
    int e = 0, e1 = 0;
    if (need) e = ar[0], e1 = ar[1];
    const int most = __reduce_max_sync(0xffffffffu, e1 - e);
    if (most <= 2)
        gather_some<2, NQ>(e, e1, amap_ent, fv, nrhs, nq, x, ab);
    else
        for (int k = 0; k < most; k += WIDE)
            gather_some<WIDE, NQ>(e + k, e1, amap_ent, fv, nrhs, nq, x, ab);
}

// Forward, task (s, i0 | cnt << 16): row tiles i0 .. i0 + cnt - 1 of front s.
// Each gathers its rows of the front vector (right-hand side on the pivot
// rows plus the children's update rows, child by child; one tile ahead) and
// accumulates acc = sum_{k < min(i, nt1)} L(i, k) y_k over the pivot tiles.
// A pivot tile (i0 < nt1, cnt = 1) then solves y_i = inv(L_ii) (f_i - acc)
// into the solution and publishes it; an update tile leaves f_i - acc in the
// front vector for the parent.  One right-hand side: r = row in the tile, the
// 64 columns of a block split over four column phases held by lanes of one
// warp (rows 8w .. 8w + 7 of warp w), so a row's sum is two shuffles.
template <typename TL>
__device__ void fwd_tile_task(int2 tk, const FrontDesc* __restrict__ fronts,
                              double* __restrict__ pub, const SolveAbort& ab,
                              const int64_t* __restrict__ fv_off,
                              const int* __restrict__ amap_off, const int* __restrict__ amap_row,
                              const int* __restrict__ amap_ent,
                              const int64_t* __restrict__ dinv_off, const TL* __restrict__ Ls,
                              const TL* __restrict__ Dinv, double* __restrict__ xp,
                              double* __restrict__ fv) {
    constexpr int T = kTile, LD = blk_ld<TL>();
    const LevelSmem<TL, false> sm;
    const int tid = threadIdx.x;
    const int r = 8 * (tid >> 5) + (tid & 7), g = (tid >> 3) & 3;
    const int s = tk.x, i0 = tk.y & 0xffff, cnt = tk.y >> 16;
    const FrontDesc F = fronts[s];
    const int nt1 = tiles_l(F.c, T);
    const bool pivot = i0 < nt1;
    const int kend = pivot ? i0 : nt1;  // L blocks per tile
    const int P = cnt * kend;
    const TL* L = Ls + F.loff;
    double* pb = pub + (dinv_off[s] / (T * T)) * T;  // this front's pivot tiles
    double* f = front_vec(fv, fv_off, s, 1);
    // the row offset of this task's blocks in their stage columns (every row
    // tile of a task starts at the same residue: 0 for a pivot tile, c for
    // update tiles)
    const int db = blk_off<TL>(tile_range(i0, F.m, F.c, T).start);
    const int aoff = amap_off[s];
    // this thread's row of tile i of the front vector (after an abort what is
    // gathered and published no longer matters, and every later wait returns)
    auto gather_row = [&](int i) -> double {
        const TileRange ti = tile_range(i, F.m, F.c, T);
        const int R = ti.start + r;
        const bool own = g == 0 && r < ti.size;
        double x[1] = {own && R < F.c ? xp[F.first_col + R] : 0.0};
        gather_entries<1>(own, amap_row + aoff + R, amap_ent, fv, 1, 1, x, ab);
        return x[0];
    };
    auto issue = [&](int p) {
        if (p < P) {
            const int i = i0 + p / kend, k = p % kend;
            const TileRange ti = tile_range(i, F.m, F.c, T);
            load_block_async(sm.lb(p), L + (int64_t)k * T * F.ldl, F.ldl, ti.start, ti.size,
                             min(T, F.c - k * T));
            load_slot_async(sm.vb(p), pb + (int64_t)k * T, 1);
        }
        cp_async_commit_group();
    };
    if (pivot) {
        const TileRange ti = tile_range(i0, F.m, F.c, T);
        load_block_async(sm.Dk, Dinv + dinv_off[s] + (int64_t)i0 * T * T, T, 0, ti.size, ti.size);
    }
    for (int p = 0; p + 1 < sm.S; ++p) issue(p);
    double fcur = gather_row(i0), acc = 0.0;
    double fnext = cnt > 1 ? gather_row(i0 + 1) : 0.0;
    bool ok = true;
    for (int p = 0; p < P; ++p) {
        issue(p + sm.S - 1);
        cp_async_wait_groups<sm.S - 1>();
        __syncthreads();
        const int i = i0 + p / kend, k = p % kend;
        double* Yk = sm.vb(p);
        if (!settle_slot(Yk, pb + (int64_t)k * T, min(T, F.c - k * T), 1, ab)) {
            ok = false;
            break;
        }
        acc += row_dot(sm.lb(p) + db + r, Yk, g);
        if (!pivot && k == kend - 1) {  // update tile i complete: f_i - acc to the front vector
            const TileRange ti = tile_range(i, F.m, F.c, T);
            double v = acc + __shfl_xor_sync(0xffffffffu, acc, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            if (g == 0 && r < ti.size) st_relaxed_f64(f + ti.start + r, fcur - v);
            acc = 0.0;
            fcur = fnext;
            if (i + 2 < i0 + cnt) fnext = gather_row(i + 2);
        }
        if (p + 1 < P) __syncthreads();  // the stages are reused; after the last, nothing is
    }
    cp_async_wait_groups<0>();
    if (!ok || !pivot) return;
    // pivot tile: F = f_i - acc (zero beyond the tile), then y = Dk F; one
    // barrier: the row's phases summed by shuffles, F into sm.Y, then y the
    // same way
    const TileRange ti = tile_range(i0, F.m, F.c, T);
    double* Y = sm.Y;
    double a = acc + __shfl_xor_sync(0xffffffffu, acc, 8);
    a += __shfl_xor_sync(0xffffffffu, a, 16);
    if (g == 0) Y[r] = r < ti.size ? fcur - a : 0.0;
    __syncthreads();
    double y = row_dot(sm.Dk + r, Y, g);
    y += __shfl_xor_sync(0xffffffffu, y, 8);
    y += __shfl_xor_sync(0xffffffffu, y, 16);
    if (g == 0 && r < ti.size) {
        xp[F.first_col + ti.start + r] = y;
        st_relaxed_f64(pb + (int64_t)i0 * T + r, y);
    }
}

// ---------------------------------------------------------------------------
// several right-hand sides: groups of up to eight, the columns of one matrix
// instruction, each group a sweep of its own inside the launch (item k of the
// list runs for every group in turn, and a group's waits, publication slots
// and front vectors are its own).  A sweep is a chain of hand-overs between
// tiles, so eight right-hand sides take about as long as one, and further
// groups run beside the first on SMs that would idle; L is read once per
// group, from L2 where the groups follow each other closely.  A warp owns
// eight rows of a 64-row block: lane (g, t) holds row 8 w + g, right-hand
// sides 2 t and 2 t + 1 (the accumulator of mma m8n8k4 over FP64).
// ---------------------------------------------------------------------------

__device__ __forceinline__ void dmma_884(double (&c)[2], double a, double b) {
    asm volatile(
        "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}
// acc += M V over 64 columns of M; M(r, k) at B[db + r + k LD] (TRANS: at
// B[db + k + r LD]), V(k, q) at V[k + q kVecLD]; two chains of accumulators
template <typename TL, bool TRANS>
__device__ __forceinline__ void group_product(const TL* B, int db, const double* V,
                                              double (&acc)[2][2]) {
    constexpr int LD = blk_ld<TL>();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r = 8 * (threadIdx.x >> 5) + g;
    const TL* Br = B + db + (TRANS ? t + r * LD : r + t * LD);
    const double* Vg = V + g * kVecLD + t;
#pragma unroll
    for (int s = 0; s < kTile / 4; ++s)
        dmma_884(acc[s & 1], (double)Br[TRANS ? 4 * s : 4 * s * LD], Vg[4 * s]);
}

// As fwd_tile_task for a group of nrhs <= 8 right-hand sides (xp, fv, pub:
// the group's own).
template <typename TL>
__device__ void fwd_tile_group(int2 tk, const FrontDesc* __restrict__ fronts,
                               double* __restrict__ pub, const SolveAbort& ab,
                               const int64_t* __restrict__ fv_off,
                               const int* __restrict__ amap_off, const int* __restrict__ amap_row,
                               const int* __restrict__ amap_ent,
                               const int64_t* __restrict__ dinv_off, const TL* __restrict__ Ls,
                               const TL* __restrict__ Dinv, double* __restrict__ xp,
                               double* __restrict__ fv, int nrhs) {
    constexpr int T = kTile;
    const LevelSmem<TL, true> sm;
    const int r = threadIdx.x >> 2, q = 2 * (threadIdx.x & 3);
    const bool q0 = q < nrhs, q1 = q + 1 < nrhs;
    const int s = tk.x, i0 = tk.y & 0xffff, cnt = tk.y >> 16;
    const FrontDesc F = fronts[s];
    const int nt1 = tiles_l(F.c, T);
    const bool pivot = i0 < nt1;
    const int kend = pivot ? i0 : nt1;  // L blocks per tile
    const int P = cnt * kend;
    const TL* L = Ls + F.loff;
    double* pb = pub + (dinv_off[s] / (T * T)) * T * nrhs;  // this front's pivot tiles
    double* f = front_vec(fv, fv_off, s, nrhs);
    const int db = blk_off<TL>(tile_range(i0, F.m, F.c, T).start);
    const int aoff = amap_off[s];
    auto gather_row = [&](int i, double (&v)[2]) {
        const TileRange ti = tile_range(i, F.m, F.c, T);
        const int R = ti.start + r;
        const bool own = r < ti.size && q0;
        v[0] = v[1] = 0.0;
        if (own && R < F.c) {
            const double* x = xp + (int64_t)(F.first_col + R) * nrhs + q;
            v[0] = x[0];
            if (q1) v[1] = x[1];
        }
        gather_entries<2>(own, amap_row + aoff + R, amap_ent, fv + q, nrhs, q1 ? 2 : 1, v, ab);
    };
    auto issue = [&](int p) {
        if (p < P) {
            const int i = i0 + p / kend, k = p % kend;
            const TileRange ti = tile_range(i, F.m, F.c, T);
            load_block_async(sm.lb(p), L + (int64_t)k * T * F.ldl, F.ldl, ti.start, ti.size,
                             min(T, F.c - k * T));
            load_slot_async(sm.vb(p), pb + (int64_t)k * T * nrhs, nrhs);
        } else if (pivot && p == P) {
            const int sz = tile_range(i0, F.m, F.c, T).size;
            load_block_async(sm.lb(p), Dinv + dinv_off[s] + (int64_t)i0 * T * T, T, 0, sz, sz);
        }
        cp_async_commit_group();
    };
    for (int p = 0; p + 1 < sm.S; ++p) issue(p);
    double fcur[2], fnext[2] = {0.0, 0.0}, acc[2][2] = {};
    gather_row(i0, fcur);
    if (cnt > 1) gather_row(i0 + 1, fnext);
    bool ok = true;
    for (int p = 0; p < P; ++p) {
        issue(p + sm.S - 1);
        cp_async_wait_groups<sm.S - 1>();
        __syncthreads();
        const int i = i0 + p / kend, k = p % kend;
        if (!settle_slot(sm.vb(p), pb + (int64_t)k * T * nrhs, min(T, F.c - k * T), nrhs, ab)) {
            ok = false;
            break;
        }
        group_product<TL, false>(sm.lb(p), db, sm.vb(p), acc);
        if (!pivot && k == kend - 1) {  // update tile i complete
            const TileRange ti = tile_range(i, F.m, F.c, T);
            if (r < ti.size) {
                double* o = f + (int64_t)(ti.start + r) * nrhs + q;
                if (q0) st_relaxed_f64(o, fcur[0] - (acc[0][0] + acc[1][0]));
                if (q1) st_relaxed_f64(o + 1, fcur[1] - (acc[0][1] + acc[1][1]));
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                acc[0][j] = acc[1][j] = 0.0;
                fcur[j] = fnext[j];
            }
            if (i + 2 < i0 + cnt) gather_row(i + 2, fnext);
        }
        if (p + 1 < P || pivot) __syncthreads();  // the stages are reused
    }
    cp_async_wait_groups<0>();
    if (!ok || !pivot) return;
    const TileRange ti = tile_range(i0, F.m, F.c, T);
    const bool in = r < ti.size;
    sm.Y[r + q * kVecLD] = in && q0 ? fcur[0] - (acc[0][0] + acc[1][0]) : 0.0;
    sm.Y[r + (q + 1) * kVecLD] = in && q1 ? fcur[1] - (acc[0][1] + acc[1][1]) : 0.0;
    __syncthreads();
    double y[2][2] = {};
    group_product<TL, false>(sm.lb(P), 0, sm.Y, y);
    if (in) {
        double* o = pb + (int64_t)i0 * nrhs * T + r;
        if (q0) {
            xp[(int64_t)(F.first_col + ti.start + r) * nrhs + q] = y[0][0] + y[1][0];
            st_relaxed_f64(o + q * T, y[0][0] + y[1][0]);
        }
        if (q1) {
            xp[(int64_t)(F.first_col + ti.start + r) * nrhs + q + 1] = y[0][1] + y[1][1];
            st_relaxed_f64(o + (q + 1) * T, y[0][1] + y[1][1]);
        }
    }
}

// Backward, update rows, task (s, j | h << 16): the partial sum
// L(k, j)' x_k over the update row tiles k of chunk h (kGatherTiles tiles;
// x final: ancestors, read through the row list) for pivot column tile j,
// published as a T x nrhs vector for the pivot task to add in chunk order.
// MULTI: a group of nrhs <= 8 right-hand sides on the matrix
// instructions; one: warp w takes columns 8w .. 8w + 7, lane (c1 = column,
// q1 = row phase) the rows q1, q1 + 4, ...: conflict-free reads of the stage
// layout, the phases summed by shuffles.
template <typename TL, bool MULTI>
__device__ void bwd_gather_task(int2 tk, const FrontDesc* __restrict__ fronts,
                                const int* __restrict__ rows, const int* __restrict__ gather_nch,
                                const int* __restrict__ gather_off, const SolveAbort& ab,
                                const TL* __restrict__ Ls, const double* __restrict__ xs,
                                double* __restrict__ part, int nrhs) {
    constexpr int T = kTile, LD = blk_ld<TL>(), GC = SolveScheduleHost::kGatherTiles;
    const LevelSmem<TL, MULTI> sm;
    const int tid = threadIdx.x;
    const int s = tk.x, j = tk.y & 0xffff, h = tk.y >> 16;
    const FrontDesc F = fronts[s];
    const int nt1 = tiles_l(F.c, T), NT = nt1 + tiles_l(F.m - F.c, T);
    const TileRange tj = tile_range(j, F.m, F.c, T);
    const TL* Lc = Ls + F.loff + (int64_t)tj.start * F.ldl;
    const int* rw = rows + F.rows_off;
    const int k0 = nt1 + h * GC, P = min(NT, k0 + GC) - k0;
    // update row tiles start at c + 64 u: one row offset for every block
    const int db = blk_off<TL>(F.c);
    const int c1 = 8 * (tid >> 5) + (tid & 7), q1 = (tid >> 3) & 3;
    // the chunk's solution rows (ancestors), then the pipeline
    for (int e = tid; e < P * T; e += blockDim.x) {
        const TileRange tkr = tile_range(k0 + e / T, F.m, F.c, T);
        const int rr = e & (T - 1);
        sm.idx[e] = rr < tkr.size ? rw[tkr.start + rr] : -1;
    }
    const int pcol = F.parent >= 0 ? fronts[F.parent].first_col : -1;
    auto issue = [&](int p) {
        if (p < P) {
            const TileRange tkr = tile_range(k0 + p, F.m, F.c, T);
            load_block_async(sm.lb(p), Lc, F.ldl, tkr.start, tkr.size, tj.size);
        }
        cp_async_commit_group();
    };
    for (int p = 0; p + 1 < sm.S; ++p) issue(p);
    if (tid < 32) await_parent(pcol, xs, nrhs, ab);
    __syncthreads();
    // the stages: the L blocks by cp.async; the ancestors' solution rows, as
    // they are published, into registers one stage ahead, stored into their
    // stage after the previous stage's products
    constexpr int VPT = MULTI ? kTile * kGroupRhs / 256 : 1;
    double pend[VPT][1];
    auto fetch = [&](int p) {
        const double* src[VPT];
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const int e = tid + 256 * k;
            const int row = p < P && e < T * nrhs ? sm.idx[p * T + (e & (T - 1))] : -1;
            src[k] = xs + (int64_t)max(row, 0) * nrhs + e / T;
            peek_values<1>(src[k], row >= 0, 1, pend[k]);
        }
        await_together<VPT, 1>([&](int k) { return src[k]; }, 1, pend, 0xffffffffu, ab);
    };
    auto put = [&](int p) {
        if (p >= P) return;
        double* v = sm.vb(p);
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const int e = tid + 256 * k;
            if (e < T * nrhs) v[(e / T) * kVecLD + (e & (T - 1))] = pend[k][0];
        }
    };
    fetch(0);
    put(0);
    double acc[2][2] = {};
    for (int p = 0; p < P; ++p) {
        issue(p + sm.S - 1);
        fetch(p + 1);
        cp_async_wait_groups<sm.S - 1>();
        __syncthreads();
        const TL* Bk = sm.lb(p);
        const double* X = sm.vb(p);
        if constexpr (MULTI) {
            group_product<TL, true>(Bk, db, X, acc);
        } else {
#pragma unroll
            for (int u = 0; u < 16; ++u)
                acc[0][0] += (double)Bk[db + q1 + 4 * u + c1 * LD] * X[q1 + 4 * u];
        }
        __syncthreads();
        put(p + 1);
    }
    cp_async_wait_groups<0>();
    double* out = part + ((int64_t)gather_off[s] + (int64_t)j * gather_nch[s] + h) * T * nrhs;
    if constexpr (MULTI) {
        const int l = tid >> 2, q = 2 * (tid & 3);
        if (q < nrhs) st_relaxed_f64(out + l + T * q, acc[0][0] + acc[1][0]);
        if (q + 1 < nrhs) st_relaxed_f64(out + l + T * (q + 1), acc[0][1] + acc[1][1]);
    } else {
        double v = acc[0][0] + __shfl_xor_sync(0xffffffffu, acc[0][0], 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (q1 == 0) st_relaxed_f64(out + c1, v);
    }
}

// ---------------------------------------------------------------------------
// small fronts: a group of W lanes per front (W = 32: fronts of up to 160
// rows, lane r holding rows r, r + 32, ... in R slots; W = 16, 8: one row per
// lane, two and four fronts per warp), the right-hand sides in passes of NQ.
// No block barriers.  Everything that does not depend on other fronts -- the
// children's places in the front vector, the first columns of L, the
// reciprocals of the pivots -- is loaded before the first wait, and the
// columns of L a chunk at a time after it: the chain from a front's children to
// its own values is one trip through L2, the assembly, and about 50 cycles per
// pivot column (a shuffle and two FP64 operations) plus a load per chunk.
// ---------------------------------------------------------------------------

template <int N>
using Int = std::integral_constant<int, N>;

template <int W>
__device__ __forceinline__ unsigned group_mask() {
    return W == 32 ? 0xffffffffu : (((1u << W) - 1u) << ((threadIdx.x & 31) & ~(W - 1)));
}

// columns of L taken at a time and the right-hand sides of a pass, by the
// registers they take (R chunk elements of L, R NQ values)
template <int R, int NQ>
constexpr int solve_chunk() {
    return R == 1 ? (NQ == 1 ? 8 : 4) : NQ == 1 ? 4 : 2;
}
template <int R, bool MULTI>
constexpr int solve_pass() {
    return !MULTI ? 1 : R == 1 ? kGroupRhs : 2;
}
// Forward.  buf: the group's shared rows, row r of right-hand side q at
// buf[32 R q + r]; rds: its reciprocals.
template <typename TL, int W, int R, int NQ>
__device__ void fwd_front(int s, const FrontDesc& F, const SolveAbort& ab,
                          const FrontDesc* __restrict__ fronts, const int* __restrict__ child,
                          const int* __restrict__ relmap, const int64_t* __restrict__ fv_off,
                          const TL* __restrict__ Ls, double* __restrict__ xp,
                          double* __restrict__ fv, int nrhs, double* buf, double* rds) {
    static_assert(W == 32 || R == 1, "several rows per lane only on whole warps");
    constexpr int stride = 32 * R;
    constexpr int CH = solve_chunk<R, NQ>(), PC = R == 1 && NQ == 1 ? 2 : 1;
    const unsigned mask = group_mask<W>();
    const int lane = threadIdx.x & (W - 1);
    const int m = F.m, c = F.c, nch = F.child_end - F.child_beg;
    const int64_t ldl = F.ldl;
    const TL* L = Ls + F.loff;
    double* out = front_vec(fv, fv_off, s, nrhs);
    for (int r = lane; r < c; r += W) rds[r] = 1.0 / (double)L[r + r * ldl];
    // PC children from the h-th on: their descriptions, then their rows' places
    // in this front.  With eight right-hand sides a pass the next child's
    // description is read under the wait for this one's values (3000 leaves under
    // a root of 8 columns, two right-hand sides FP32: 2.3 ms; read after it 3.2)
    constexpr bool AHEAD = R == 1 && NQ == kGroupRhs;
    int d_c[PC], d_uc[PC], d_rows[PC];
    int64_t d_fv[PC];
    auto describe = [&](int h) {
#pragma unroll
        for (int e = 0; e < PC; ++e) {
            const bool has = h + e < nch;
            const int ch = has ? child[F.child_beg + h + e] : s;
            d_c[e] = fronts[ch].c;
            d_uc[e] = has ? fronts[ch].m - d_c[e] : 0;
            d_rows[e] = fronts[ch].rows_off + d_c[e];
            d_fv[e] = fv_off[ch];
        }
    };
    int pc[PC][R];
    const double* wp[PC];
    auto places = [&]() {
#pragma unroll
        for (int e = 0; e < PC; ++e) {
            wp[e] = fv + (d_fv[e] + d_c[e]) * nrhs;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int r = lane + W * k;
                pc[e][k] = -1;
                if (r < d_uc[e]) pc[e][k] = relmap[d_rows[e] + r];
            }
        }
    };
    TL l[R][CH];
    auto columns = [&](int j0) {
#pragma unroll
        for (int cc = 0; cc < CH; ++cc)
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int r = lane + W * k, j = j0 + cc;
                l[k][cc] = TL(0);
                if (r > j && r < m && j < c) l[k][cc] = L[r + j * ldl];
            }
    };
    describe(0);
    places();
    for (int q0 = 0; q0 < nrhs; q0 += NQ) {
        const int nq = min(NQ, nrhs - q0);
        columns(0);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int r = lane + W * k;
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (r < m && q < nq)
                    buf[q * stride + r] =
                        r < c ? xp[(int64_t)(F.first_col + r) * nrhs + q0 + q] : 0.0;
        }
        __syncwarp(mask);
        for (int h = 0; h < nch; h += PC) {  // children in order
            if (h > 0 || (q0 > 0 && nch > PC)) {
                if (!AHEAD || h == 0) describe(h);
                places();
            }
            double w[PC][R][NQ];
            auto at = [&](int e, int k) { return wp[e] + (int64_t)(lane + W * k) * nrhs + q0; };
#pragma unroll
            for (int e = 0; e < PC; ++e)
#pragma unroll
                for (int k = 0; k < R; ++k) peek_values<NQ>(at(e, k), pc[e][k] >= 0, nq, w[e][k]);
            if (AHEAD && h + PC < nch) describe(h + PC);
#pragma unroll
            for (int e = 0; e < PC; ++e) {
                await_together<R, NQ>([&](int k) { return at(e, k); }, nq, w[e], mask, ab);
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    if (pc[e][k] >= 0)
#pragma unroll
                        for (int q = 0; q < NQ; ++q)
                            if (q < nq) buf[q * stride + pc[e][k]] += w[e][k][q];
                }
                __syncwarp(mask);
            }
        }
        double v[R][NQ];
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                v[k][q] = (q < nq && lane + W * k < m) ? buf[q * stride + lane + W * k] : 0.0;
        __syncwarp(mask);
#pragma unroll
        for (int ks = 0; ks < R; ++ks) {  // pivot columns W ks .. W ks + W - 1
            for (int j0 = W * ks; j0 < min(c, W * (ks + 1)); j0 += CH) {
                if (j0 > 0) columns(j0);
#pragma unroll
                for (int cc = 0; cc < CH; ++cc) {
                    const int j = j0 + cc - W * ks;  // the pivot's lane
                    if (j0 + cc >= c) break;
                    const double rj = rds[j0 + cc];
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        const double y = __shfl_sync(mask, v[ks][q], j, W) * rj;
#pragma unroll
                        for (int k = ks; k < R; ++k)
                            if (NQ > 1 || k > ks || lane > j) v[k][q] -= (double)l[k][cc] * y;
                        if (lane == j) v[ks][q] = y;
                    }
                }
            }
        }
        // Several right-hand sides (a test per column cost them 4 to 9 %, one
        // right-hand side nothing): an infinite y left 0 y, a NaN, on the rows
        // above its pivot.  The front again from its assembled rows, column by
        // column in shared memory, the rows below a pivot only.
        double z = 0.0;
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
            for (int q = 0; q < NQ; ++q) z = fma(v[k][q], 0.0, z);
        if (NQ > 1 && __any_sync(mask, z != 0.0)) {
            for (int j = 0; j < c; ++j)
                for (int q = 0; q < nq; ++q) {
                    double* b = buf + q * stride;
                    const double y = b[j] * rds[j];
                    __syncwarp(mask);
                    for (int r = j + lane; r < m; r += W)
                        b[r] = r == j ? y : b[r] - (double)L[r + j * ldl] * y;
                    __syncwarp(mask);
                }
#pragma unroll
            for (int k = 0; k < R; ++k)
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    if (q < nq && lane + W * k < m) v[k][q] = buf[q * stride + lane + W * k];
        }
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int r = lane + W * k;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                if (q >= nq || r >= m) continue;
                if (r < c)
                    xp[(int64_t)(F.first_col + r) * nrhs + q0 + q] = v[k][q];
                else
                    st_relaxed_f64(out + r * nrhs + q0 + q, v[k][q]);
            }
        }
    }
}

// Backward: t = y - L21' x over the update rows (one reduction per pivot column,
// independent of each other), then the pivot columns from the last, lane i
// holding column i: x_j = t_j / L(j, j), t_i -= L(j, i) x_j, the rows j
// of L read four at a time down each lane's own column.
template <typename TL, int W, int R, int NQ>
__device__ void bwd_front(const FrontDesc& F, const SolveAbort& ab,
                          const FrontDesc* __restrict__ fronts, const int* __restrict__ rows,
                          const TL* __restrict__ Ls, const double* __restrict__ xp,
                          double* __restrict__ xs, int nrhs, double* rds) {
    static_assert(W == 32 || R == 1, "several rows per lane only on whole warps");
    constexpr int CH = NQ == 8 ? 1 : solve_chunk<R, NQ>();
    const unsigned mask = group_mask<W>();
    const int lane = threadIdx.x & (W - 1);
    const int m = F.m, c = F.c;
    const int64_t ldl = F.ldl;
    const TL* L = Ls + F.loff;
    int src[R];  // this lane's update rows in the solution
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int r = lane + W * k;
        src[k] = -1;
        if (r >= c && r < m) src[k] = rows[F.rows_off + r];
    }
    for (int r = lane; r < c; r += W) rds[r] = 1.0 / (double)L[r + r * ldl];
    __syncwarp(mask);
    TL l[R][CH];
    auto columns = [&](int j0) {
#pragma unroll
        for (int cc = 0; cc < CH; ++cc)
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int r = lane + W * k;
                l[k][cc] = TL(0);
                if (r >= c && r < m && j0 + cc < c) l[k][cc] = L[r + (j0 + cc) * ldl];
            }
    };
    // rows 4 b .. 4 b + 3 of L in column lane + W k
    TL lt[R][4];
    auto pivot_rows = [&](int b) {
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int i = lane + W * k;
#pragma unroll
            for (int e = 0; e < 4; ++e) lt[k][e] = TL(0);
            if (i < c && i < 4 * b + 4) ld4(L + 4 * b + i * ldl, lt[k]);
        }
    };
    for (int q0 = 0; q0 < nrhs; q0 += NQ) {
        const int nq = min(NQ, nrhs - q0);
        double t[R][NQ], x[R][NQ];
        columns(0);
        if (R == 1) pivot_rows((c - 1) / 4);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int r = lane + W * k;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                t[k][q] = 0.0;
                if (r < c && q < nq)
                    t[k][q] = xp[(int64_t)(F.first_col + r) * nrhs + q0 + q];
            }
        }
#pragma unroll
        for (int k = 0; k < R; ++k)
            peek_values<NQ>(xs + (int64_t)max(src[k], 0) * nrhs + q0, src[k] >= 0, nq, x[k]);
        await_together<R, NQ>([&](int k) { return xs + (int64_t)max(src[k], 0) * nrhs + q0; }, nq,
                              x, mask, ab);
        if (m > c) {
#pragma unroll
            for (int ks = 0; ks < R; ++ks) {
                for (int j0 = W * ks; j0 < min(c, W * (ks + 1)); j0 += CH) {
                    if (j0 > 0) columns(j0);
                    double p[CH][NQ];
#pragma unroll
                    for (int cc = 0; cc < CH; ++cc)
#pragma unroll
                        for (int q = 0; q < NQ; ++q) {
                            p[cc][q] = 0.0;
#pragma unroll
                            for (int k = 0; k < R; ++k) p[cc][q] += (double)l[k][cc] * x[k][q];
                        }
#pragma unroll
                    for (int o = W / 2; o > 0; o >>= 1)
#pragma unroll
                        for (int cc = 0; cc < CH; ++cc)
#pragma unroll
                            for (int q = 0; q < NQ; ++q)
                                p[cc][q] += __shfl_xor_sync(mask, p[cc][q], o, W);
#pragma unroll
                    for (int cc = 0; cc < CH; ++cc)
#pragma unroll
                        for (int q = 0; q < NQ; ++q)
                            if (lane == j0 + cc - W * ks) t[ks][q] -= p[cc][q];
                }
            }
        }
#pragma unroll
        for (int ks = R - 1; ks >= 0; --ks) {
            for (int b = (min(c, W * (ks + 1)) - 1) / 4; b >= W * ks / 4; --b) {
                if (R > 1 || 4 * b + 4 < c) pivot_rows(b);
#pragma unroll
                for (int e = 3; e >= 0; --e) {
                    const int j = 4 * b + e;
                    if (j >= c) continue;
                    const double rj = rds[j];
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        const double xj = __shfl_sync(mask, t[ks][q], j - W * ks, W) * rj;
#pragma unroll
                        for (int k = 0; k <= ks; ++k)
                            if (lane + W * k < j) t[k][q] -= (double)lt[k][e] * xj;
                        if (lane == j - W * ks) t[ks][q] = xj;
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int r = lane + W * k;
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (q < nq && r < c)
                    st_relaxed_f64(xs + (int64_t)(F.first_col + r) * nrhs + q0 + q, t[k][q]);
        }
    }
}

// per-warp shared buffer of the small fronts: the reciprocals of the pivots,
// then the rows of a pass (32 R rows of solve_pass() right-hand sides)
constexpr int kWarpBufRows = ((Plan::kSmallMaxRows + 31) / 32) * 32;
template <bool MULTI>
__host__ __device__ constexpr int warp_buf() {
    return kWarpBufRows + (MULTI ? 32 * 12 : kWarpBufRows);
}
static_assert(32 * solve_pass<1, true>() <= 32 * 12 && 32 * 5 * solve_pass<5, true>() <= 32 * 12,
              "a pass of either kind fits the buffer");

// Warp tasks of one warp item (its slice of the direction's warp list):
// tasks [0, n1) one front each, then two fronts of 9..16 rows per task, then
// four of at most 8 rows.
struct WarpTasks {
    const int* list;
    int n1, n2, n4;
    __host__ __device__ int count() const { return n1 + (n2 + 1) / 2 + (n4 + 3) / 4; }
};


template <typename TL, bool MULTI>
__device__ void fwd_warp_task(const WarpTasks& wt, int t, const SolveAbort& ab,
                              const FrontDesc* __restrict__ fronts,
                              const int* __restrict__ child, const int* __restrict__ relmap,
                              const int64_t* __restrict__ fv_off, const TL* __restrict__ Ls,
                              double* __restrict__ xp, double* __restrict__ fv, int nrhs,
                              double* wbuf) {
    const int lane = threadIdx.x & 31, t2 = (wt.n2 + 1) / 2;
    auto front = [&](auto w, auto r, int s) {
        const FrontDesc F = fronts[s];
        constexpr int W = decltype(w)::value, R = decltype(r)::value;
        const int g = W < 32 ? lane & ~(W - 1) : 0;  // the group's place in the buffer
        fwd_front<TL, W, R, solve_pass<R, MULTI>()>(s, F, ab, fronts, child, relmap, fv_off, Ls,
                                                    xp, fv, nrhs, wbuf + kWarpBufRows + g,
                                                    wbuf + g);
    };
    if (t < wt.n1) {
        const int s = wt.list[t];
        const int m = fronts[s].m;
        if (m <= 32) front(Int<32>(), Int<1>(), s);
        else front(Int<32>(), Int<5>(), s);
    } else if ((t -= wt.n1) < t2) {
        const int k = 2 * t + (lane >> 4);
        if (k < wt.n2) front(Int<16>(), Int<1>(), wt.list[wt.n1 + k]);
    } else {
        const int k = 4 * (t - t2) + (lane >> 3);
        if (k < wt.n4) front(Int<8>(), Int<1>(), wt.list[wt.n1 + wt.n2 + k]);
    }
}

template <typename TL, bool MULTI>
__device__ void bwd_warp_task(const WarpTasks& wt, int t, const SolveAbort& ab,
                              const FrontDesc* __restrict__ fronts, const int* __restrict__ rows,
                              const TL* __restrict__ Ls, const double* __restrict__ xp,
                              double* __restrict__ xs, int nrhs, double* wbuf) {
    const int lane = threadIdx.x & 31, t2 = (wt.n2 + 1) / 2;
    auto front = [&](auto w, auto r, int s) {
        const FrontDesc F = fronts[s];
        constexpr int W = decltype(w)::value, R = decltype(r)::value;
        bwd_front<TL, W, R, solve_pass<R, MULTI>()>(F, ab, fronts, rows, Ls, xp, xs, nrhs,
                                                    wbuf + (W < 32 ? lane & ~(W - 1) : 0));
    };
    if (t < wt.n1) {
        const int s = wt.list[t];
        const int m = fronts[s].m;
        if (m <= 32) front(Int<32>(), Int<1>(), s);
        else front(Int<32>(), Int<5>(), s);
    } else if ((t -= wt.n1) < t2) {
        const int k = 2 * t + (lane >> 4);
        if (k < wt.n2) front(Int<16>(), Int<1>(), wt.list[wt.n1 + k]);
    } else {
        const int k = 4 * (t - t2) + (lane >> 3);
        if (k < wt.n4) front(Int<8>(), Int<1>(), wt.list[wt.n1 + wt.n2 + k]);
    }
}

// Backward, task (s, j): pivot column tile j of front s accumulates the
// partial sums of the update-row gathers of (s, j), as they are published, in
// chunk order, then acc += sum_{k > j} L(k, j)' x_k over the pivot tiles
// nt1-1 .. j+1 of this front as they publish, and solves
// x_j = inv(L_jj)' (y_j - acc).  MULTI as in bwd_gather_task.
template <typename TL, bool MULTI>
__device__ void bwd_chain_task(int2 tk, const FrontDesc* __restrict__ fronts,
                               double* __restrict__ pub, const SolveAbort& ab,
                               const int* __restrict__ gather_nch,
                               const int* __restrict__ gather_off,
                               const double* __restrict__ part,
                               const int64_t* __restrict__ dinv_off, const TL* __restrict__ Ls,
                               const TL* __restrict__ Dinv, const double* __restrict__ xp,
                               double* __restrict__ xs, int nrhs) {
    constexpr int T = kTile, LD = blk_ld<TL>();
    const LevelSmem<TL, MULTI> sm;
    const int tid = threadIdx.x;
    // this thread's column of the tile and right-hand sides: several, two of
    // column tid / 4; one, phase 0 of column c1
    const int q1 = (tid >> 3) & 3;
    const int l = MULTI ? tid >> 2 : 8 * (tid >> 5) + (tid & 7), q = MULTI ? 2 * (tid & 3) : 0;
    const bool own0 = MULTI ? q < nrhs : q1 == 0, own1 = MULTI && q + 1 < nrhs;
    const int s = tk.x, j = tk.y;
    const FrontDesc F = fronts[s];
    const int nt1 = tiles_l(F.c, T);
    const TileRange tj = tile_range(j, F.m, F.c, T);
    const TL* Lc = Ls + F.loff + (int64_t)tj.start * F.ldl;  // column tile j
    const int64_t tile0 = dinv_off[s] / (T * T);               // this front's first pivot tile
    double* pb = pub + tile0 * T * nrhs;
    const int P = nt1 - 1 - j;  // pivot row tiles k = nt1-1 down to j+1
    auto load_inv = [&](TL* dst) {
        load_block_async(dst, Dinv + dinv_off[s] + (int64_t)j * T * T, T, 0, tj.size, tj.size);
    };
    auto issue = [&](int p) {
        if (p < P) {
            const TileRange tkr = tile_range(nt1 - 1 - p, F.m, F.c, T);
            load_block_async(sm.lb(p), Lc, F.ldl, tkr.start, tkr.size, tj.size);
            load_slot_async(sm.vb(p), pb + (int64_t)(nt1 - 1 - p) * T * nrhs, nrhs);
        } else if (MULTI && p == P) {
            load_inv(sm.lb(p));
        }
        cp_async_commit_group();
    };
    if (!MULTI) load_inv(sm.Dk);
    for (int p = 0; p + 1 < sm.S; ++p) issue(p);
    double acc[2][2] = {};
    // this tile's y_j, before the first wait
    const int64_t xj = F.first_col + tj.start + l;
    const bool in = l < tj.size;
    const double y0 = in && own0 ? xp[xj * nrhs + q] : 0.0;
    const double y1 = in && own1 ? xp[xj * nrhs + q + 1] : 0.0;
    // the update-row partial sums of (s, j) (gathers hold lower tickets), in
    // chunk order, before the chain's first wait; two in flight
    {
        const int nch = gather_nch[s];
        constexpr int NP = MULTI ? 2 : 1;
        const double* pj = part + ((int64_t)gather_off[s] + (int64_t)j * nch) * T * nrhs + l + T * q;
        for (int h = 0; h < nch; h += 2) {
            double v[2 * NP][1];
            auto at = [&](int k) { return pj + (int64_t)(h + k / NP) * T * nrhs + T * (k % NP); };
#pragma unroll
            for (int k = 0; k < 2 * NP; ++k)
                peek_values<1>(at(k), (k % NP == 0 ? own0 : own1) && h + k / NP < nch, 1, v[k]);
            await_together<2 * NP, 1>(at, 1, v, 0xffffffffu, ab);
#pragma unroll
            for (int k = 0; k < 2 * NP; ++k) acc[0][k % NP] += v[k][0];
        }
    }
    bool ok = true;
    for (int p = 0; p < P; ++p) {
        issue(p + sm.S - 1);
        cp_async_wait_groups<sm.S - 1>();
        __syncthreads();
        const int k = nt1 - 1 - p;
        double* X = sm.vb(p);
        if (!settle_slot(X, pb + (int64_t)k * T * nrhs, tile_range(k, F.m, F.c, T).size, nrhs, ab)) {
            ok = false;
            break;
        }
        const TL* B = sm.lb(p);
        if constexpr (MULTI) {
            group_product<TL, true>(B, 0, X, acc);
        } else {
#pragma unroll
            for (int u = 0; u < 16; ++u)
                acc[0][0] += (double)B[q1 + 4 * u + l * LD] * X[q1 + 4 * u];
        }
        if (p + 1 < P || MULTI) __syncthreads();  // the stages are reused
    }
    cp_async_wait_groups<0>();
    if (!ok) return;
    double* X = sm.Y;
    // t = y_j - acc (y_j: this front's forward solution), then x_j = Dk' t
    if constexpr (MULTI) {
        X[l + q * kVecLD] = in && own0 ? y0 - (acc[0][0] + acc[1][0]) : 0.0;
        X[l + (q + 1) * kVecLD] = in && own1 ? y1 - (acc[0][1] + acc[1][1]) : 0.0;
        __syncthreads();
        double x[2][2] = {};
        group_product<TL, true>(sm.lb(P), 0, X, x);
        if (in && own0) {
            st_relaxed_f64(xs + xj * nrhs + q, x[0][0] + x[1][0]);
            st_relaxed_f64(pb + ((int64_t)j * nrhs + q) * T + l, x[0][0] + x[1][0]);
        }
        if (in && own1) {
            st_relaxed_f64(xs + xj * nrhs + q + 1, x[0][1] + x[1][1]);
            st_relaxed_f64(pb + ((int64_t)j * nrhs + q + 1) * T + l, x[0][1] + x[1][1]);
        }
    } else {
        // one right-hand side, one barrier: the row phases' sums by
        // shuffles, t into sm.Y, then x_j = Dk' t the same way
        const TL* Dk = sm.Dk;
        double a = acc[0][0] + __shfl_xor_sync(0xffffffffu, acc[0][0], 8);
        a += __shfl_xor_sync(0xffffffffu, a, 16);
        if (q1 == 0) X[l] = in ? y0 - a : 0.0;
        __syncthreads();
        double x = 0.0;
#pragma unroll
        for (int u = 0; u < 16; ++u) x += (double)Dk[q1 + 4 * u + l * LD] * X[q1 + 4 * u];
        x += __shfl_xor_sync(0xffffffffu, x, 8);
        x += __shfl_xor_sync(0xffffffffu, x, 16);
        if (q1 == 0 && in) {
            st_relaxed_f64(pb + (int64_t)j * T + l, x);
            st_relaxed_f64(xs + xj, x);
        }
    }
}

// ---------------------------------------------------------------------------
// forward update tiles with one right-hand side: L read straight from global
// memory into registers, coalesced (a thread per row), the next columns'
// loads issued before the current ones are used, no block barrier per L
// block.  For fronts of one pivot tile, whose published vector comes through
// poll_published into shared memory (with more tiles, one column group of loads
// in flight per iteration leaves a tail of one memory latency per 16 columns
// after the last pivot tile, where the staged tile path keeps two 64-column
// blocks in flight).
// ---------------------------------------------------------------------------

// Forward update rows [R0, R1) of front s (at most 256; one right-hand side):
// thread = row; columns in groups of 16, the next group's loads issued
// before the current group's products.
template <typename TL>
__device__ void fwd_update_rt1(int s, int R0, int R1, const FrontDesc& F, double* __restrict__ pb,
                               const SolveAbort& ab, const int* __restrict__ amap_off,
                               const int* __restrict__ amap_row,
                               const int* __restrict__ amap_ent, const TL* __restrict__ Ls,
                               double* __restrict__ f, const double* __restrict__ fv) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* Y = reinterpret_cast<double*>(smem_raw);  // the pivot tile's values
    const int R = R0 + threadIdx.x;
    const bool rv = R < R1;
    const TL* Lr = Ls + F.loff + R;
    constexpr int GW = sizeof(TL) == 4 ? 16 : 8;  // columns per group (registers)
    const int ng = (F.c + GW - 1) / GW;
    auto load = [&](int cg, TL (&v)[GW]) {
#pragma unroll
        for (int l = 0; l < GW; ++l) {
            const int col = GW * cg + l;
            v[l] = (rv && col < F.c) ? __ldg(Lr + (int64_t)col * F.ldl) : TL(0);
        }
    };
    double acc = 0.0;
    TL lv[GW], ln[GW];
    load(0, lv);
    double f0[1] = {0.0};
    gather_entries<1>(rv, amap_row + amap_off[s] + R, amap_ent, fv, 1, 1, f0, ab);
    for (int cg = 0; cg < ng; ++cg) {
        if (cg + 1 < ng) load(cg + 1, ln);
        if (cg == 0 && !poll_published(Y, pb, F.c, 1, ab)) return;
        const double* y = Y + GW * cg;
#pragma unroll
        for (int l = 0; l < GW; ++l) acc += (double)lv[l] * y[l];
#pragma unroll
        for (int l = 0; l < GW; ++l) lv[l] = ln[l];
    }
    if (rv) st_relaxed_f64(f + R, f0[0] - acc);
}

// One launch per direction over all work items (the item lists, in a
// topological order by critical-path priority, and their kinds are
// described with the solve schedule): persistent CTAs take items by atomic
// ticket.  An item only waits for values that items with lower tickets
// publish -- children's (forward) and parents' (backward) items come earlier
// in the list, and so do a front's earlier pivot tiles and its backward
// gathers -- and a CTA takes a ticket only while it runs, so every wait is for
// a CTA that is running or done.  Every wait polls with an iteration limit; on
// timeout the launch is aborted (every later wait returns at once) and the
// error word reaches the host.

// Right-hand sides of a launch in groups, with the groups' slices of the work
// vectors.
struct SolveGroups {
    int n, nrhs;       // unknowns, right-hand sides of the launch
    int64_t fv_total;  // work vector rows
    // (a group's right-hand sides and solution: rows of size(g) values)
    __device__ int count() const { return nrhs == 1 ? 1 : (nrhs + kGroupRhs - 1) / kGroupRhs; }
    __device__ int size(int g) const { return min(kGroupRhs, nrhs - kGroupRhs * g); }
    __device__ int64_t xp_off(int g) const { return (int64_t)kGroupRhs * g * n; }
    __device__ int64_t fv_off(int g) const { return kGroupRhs * fv_total * g; }
};

// residency by shared memory: one right-hand side keeps the stages' blocks of L
// and an inverse per CTA (FP32 four blocks, 72 KB, FP64 three, 107 KB), a group
// two and its vectors (49 and 84 KB); by registers (the small fronts' columns of L): three CTAs
template <typename TL>
constexpr int solve_ctas_per_sm() {
    return sizeof(TL) == 8 ? 2 : 3;
}

template <typename TL, bool MULTI>
__global__ void __launch_bounds__(256, solve_ctas_per_sm<TL>())
    k_fwd_solve(const FrontDesc* __restrict__ fronts, const int4* __restrict__ items, int nitems,
                int* __restrict__ counter, int64_t pub_rows, SolveAbort ab,
                const int64_t* __restrict__ fv_off, const int* __restrict__ amap_off,
                const int* __restrict__ amap_row, const int* __restrict__ amap_ent,
                const int64_t* __restrict__ dinv_off, const int* __restrict__ wlist,
                const int* __restrict__ child,
                const int* __restrict__ relmap, const TL* __restrict__ Ls,
                const TL* __restrict__ Dinv, double* __restrict__ xp0, double* __restrict__ fv0,
                SolveGroups grp) {
    constexpr int T = kTile;
    __shared__ int s_item;
    const int ngroups = MULTI ? grp.count() : 1;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
        __syncthreads();
        const int k = s_item;
        if (k >= nitems * ngroups) return;
        const int4 it = items[MULTI ? k / ngroups : k];
        const int gi = MULTI ? k % ngroups : 0, nrhs = MULTI ? grp.size(gi) : 1;
        double* xp = xp0 + grp.xp_off(gi);
        double* fv = fv0 + grp.fv_off(gi);
        double* pub = fv + pub_rows * nrhs;
        if (it.x == SolveScheduleHost::kItemWarps) {
            extern __shared__ __align__(16) unsigned char smem_raw[];
            const WarpTasks wt{wlist + it.y, it.z & 0xff, (it.z >> 8) & 0xff, it.z >> 16};
            const int w = threadIdx.x >> 5, t = w;
            double* wbuf = reinterpret_cast<double*>(smem_raw) + w * warp_buf<MULTI>();
            if (t < wt.count())
                fwd_warp_task<TL, MULTI>(wt, t, ab, fronts, child, relmap, fv_off, Ls, xp, fv,
                                         nrhs, wbuf);
        } else {
            const int2 tk = make_int2(it.y, it.z);
            if constexpr (MULTI) {
                fwd_tile_group<TL>(tk, fronts, pub, ab, fv_off, amap_off, amap_row, amap_ent,
                                   dinv_off, Ls, Dinv, xp, fv, nrhs);
            } else {
                const int s = tk.x, i0 = tk.y & 0xffff, cnt = tk.y >> 16;
                const FrontDesc F = fronts[s];
                const int nt1 = tiles_l(F.c, T);
                if (i0 >= nt1 && nt1 == 1) {
                    // update tiles of fronts of one pivot tile, one right-hand
                    // side: registers straight from L (measured faster there;
                    // the staged pipeline streams long column ranges better)
                    double* pb = pub + (dinv_off[s] / (T * T)) * T;
                    const TileRange a = tile_range(i0, F.m, F.c, T);
                    const TileRange b = tile_range(i0 + cnt - 1, F.m, F.c, T);
                    fwd_update_rt1<TL>(s, a.start, b.start + b.size, F, pb, ab, amap_off,
                                       amap_row, amap_ent, Ls, front_vec(fv, fv_off, s, 1), fv);
                } else {
                    fwd_tile_task<TL>(tk, fronts, pub, ab, fv_off, amap_off, amap_row, amap_ent,
                                      dinv_off, Ls, Dinv, xp, fv);
                }
            }
        }
        __syncthreads();  // shared memory and s_item free for the next item
    }
}

// xs (at fv0): the solution, row k's right-hand sides side by side
template <typename TL, bool MULTI>
__global__ void __launch_bounds__(256, solve_ctas_per_sm<TL>())
    k_bwd_solve(const FrontDesc* __restrict__ fronts, const int4* __restrict__ items, int nitems,
                int* __restrict__ counter, int64_t pub_rows, int64_t part_rows, SolveAbort ab,
                const int* __restrict__ gather_nch, const int* __restrict__ gather_off,
                const int64_t* __restrict__ dinv_off, const int* __restrict__ wlist,
                const int* __restrict__ rows, const TL* __restrict__ Ls,
                const TL* __restrict__ Dinv, const double* __restrict__ xp0,
                double* __restrict__ fv0, SolveGroups grp) {
    __shared__ int s_item;
    const int ngroups = MULTI ? grp.count() : 1;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
        __syncthreads();
        const int k = s_item;
        if (k >= nitems * ngroups) return;
        const int4 it = items[MULTI ? k / ngroups : k];
        const int gi = MULTI ? k % ngroups : 0, nrhs = MULTI ? grp.size(gi) : 1;
        const double* xp = xp0 + grp.xp_off(gi);
        double* xs = fv0 + grp.fv_off(gi);
        double* pub = xs + pub_rows * nrhs;
        double* part = xs + part_rows * nrhs;
        if (it.x == SolveScheduleHost::kItemWarps) {
            const WarpTasks wt{wlist + it.y, it.z & 0xff, (it.z >> 8) & 0xff, it.z >> 16};
            extern __shared__ __align__(16) unsigned char smem_raw[];
            const int t = threadIdx.x >> 5;
            if (t < wt.count())
                bwd_warp_task<TL, MULTI>(wt, t, ab, fronts, rows, Ls, xp, xs, nrhs,
                                         reinterpret_cast<double*>(smem_raw) + t * kWarpBufRows);
        } else if (it.x == SolveScheduleHost::kItemGather) {
            bwd_gather_task<TL, MULTI>(make_int2(it.y, it.z), fronts, rows, gather_nch, gather_off,
                                       ab, Ls, xs, part, nrhs);
        } else {
            bwd_chain_task<TL, MULTI>(make_int2(it.y, it.z), fronts, pub, ab, gather_nch,
                                      gather_off, part, dinv_off, Ls, Dinv, xp, xs, nrhs);
        }
        __syncthreads();  // shared memory and s_item free for the next item
    }
}

// `rows` rows of every group's work vectors set to the unpublished pattern;
// sync (may be null): the ticket counters and the abort word cleared
__global__ void __launch_bounds__(256)
    k_solve_init(int4* __restrict__ sync, double* __restrict__ fv0, int64_t rows,
                 SolveGroups grp) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * blockDim.x;
    if (sync && tid == 0) *sync = make_int4(0, 0, 0, 0);
    const double v = __longlong_as_double(-1ll);
    for (int g = 0; g < grp.count(); ++g) {
        double* p = fv0 + grp.fv_off(g);  // on 16 bytes
        const int64_t cnt = rows * grp.size(g);
        for (int64_t i = tid; 2 * i + 1 < cnt; i += nt)
            reinterpret_cast<double2*>(p)[i] = make_double2(v, v);
        if ((cnt & 1) && tid == 0) p[cnt - 1] = v;
    }
}

// ---------------------------------------------------------------------------
// permutations
// ---------------------------------------------------------------------------

// b into groups of right-hand sides one after another, a row's right-hand
// sides of a group side by side
__global__ void k_perm_gather(const int* __restrict__ perm, const double* __restrict__ b,
                              double* __restrict__ xp, SolveGroups grp, int ldb) {
    const int n = grp.n;
    const int64_t total = (int64_t)n * grp.nrhs;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int q = (int)(idx / n), k = (int)(idx - (int64_t)q * n);
        const int g = grp.nrhs == 1 ? 0 : q / kGroupRhs;
        xp[grp.xp_off(g) + (int64_t)k * grp.size(g) + q - g * kGroupRhs] =
            b[(perm ? perm[k] : k) + (int64_t)q * ldb];
    }
}

// xs: the backward sweep's solution, groups of right-hand sides one after
// another, fv_total rows apart, a row's right-hand sides side by side
__global__ void k_perm_scatter(const int* __restrict__ perm, const double* __restrict__ xs,
                               double* __restrict__ x, SolveGroups grp, int ldx) {
    const int n = grp.n;
    const int64_t total = (int64_t)n * grp.nrhs;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int q = (int)(idx / n), k = (int)(idx - (int64_t)q * n);
        const int g = grp.nrhs == 1 ? 0 : q / kGroupRhs;
        x[(perm ? perm[k] : k) + (int64_t)q * ldx] =
            xs[grp.fv_off(g) + (int64_t)k * grp.size(g) + q - g * kGroupRhs];
    }
}

void permute_gather(const int* perm, const double* b, double* xp, int n, int nrhs, int ldb,
                    cudaStream_t st) {
    int64_t total = (int64_t)n * nrhs;
    int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 16);
    k_perm_gather<<<blocks, 256, 0, st>>>(perm, b, xp, SolveGroups{n, nrhs, 0}, ldb);
}

void permute_solution(const DevPlan& D, const int* perm, const double* fv, double* x, int nrhs,
                      int ldx, cudaStream_t st) {
    const int64_t total = (int64_t)D.n * nrhs;
    const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 16);
    k_perm_scatter<<<blocks, 256, 0, st>>>(perm, fv, x, SolveGroups{D.n, nrhs, D.fv_total}, ldx);
}

// ---------------------------------------------------------------------------
// launch sequence
// ---------------------------------------------------------------------------

// dynamic shared memory of a solve launch: the tile tasks' stages or the
// eight warps' buffers, whichever is larger
template <typename TL, bool MULTI>
static size_t solve_smem() {
    size_t m = level_smem_bytes<TL, MULTI>();
    return std::max(m, 8 * (size_t)warp_buf<MULTI>() * sizeof(double));
}

template <typename TL, bool MULTI>
static void set_solve_attributes() {
    const int sm = (int)solve_smem<TL, MULTI>();
    cudaFuncSetAttribute(k_fwd_solve<TL, MULTI>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_bwd_solve<TL, MULTI>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
}

void init_solve_kernels() {
    set_solve_attributes<double, false>();
    set_solve_attributes<float, false>();
    set_solve_attributes<double, true>();
    set_solve_attributes<float, true>();
}

template <typename TL, bool MULTI>
static void solve_launch(const DevPlan& D, const TL* Ls, const TL* Dinv, double* xp, double* fv,
                         int nrhs, cudaStream_t st) {
    const SolveSchedule& S = D.solve;
    static_assert(Plan::kSmallMaxRows <= 32 * 5, "the warp path holds 160 rows in registers");
    // sync: the two ticket counters and the abort word
    const SolveAbort ab{S.sync + 2, S.err};
    const SolveGroups grp{D.n, nrhs, D.fv_total};
    const int64_t slots = (int64_t)S.nflags * kTile;  // rows of one direction
    const int sms = D.num_sms > 0 ? D.num_sms : 148;
    auto init = [&](int4* sync, int64_t rows) {
        const int64_t work = rows * nrhs / 2;
        const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((work + 511) / 512, sms * 8));
        k_solve_init<<<blocks, 256, 0, st>>>(sync, fv, rows, grp);
    };
    const size_t sm = solve_smem<TL, MULTI>();
    const int grid = sms * solve_ctas_per_sm<TL>();
    const int ng = MULTI ? (nrhs + kGroupRhs - 1) / kGroupRhs : 1;
    double fbytes = 0, bbytes = 0;
    for (int l = 0; l < D.nlevels; ++l) {
        fbytes += (S.small_elems[l] + S.fwd_elems[l]) * sizeof(TL);
        bbytes += (S.small_elems[l] + S.bwd_elems[l]) * sizeof(TL);
    }
    init(reinterpret_cast<int4*>(S.sync), D.fv_total);
    if (S.nfwd_items > 0) {
        ProfScope ps(D.prof, KC_SOLVE_LARGE, st, 0, fbytes);
        k_fwd_solve<TL, MULTI><<<std::min(grid, S.nfwd_items * ng), 256, sm, st>>>(
            D.fronts, S.fwd_items, S.nfwd_items, S.sync, D.fv_pub_off, ab, D.fv_off, S.amap_off,
            S.amap_row, S.amap_ent, D.dinv_off, S.fwd_wlist, D.child, D.relmap, Ls, Dinv, xp, fv,
            grp);
    }
    // the solution takes the place of the front vectors (at least n rows)
    init(nullptr, D.n);
    if (S.nbwd_items > 0) {
        ProfScope ps(D.prof, KC_SOLVE_LARGE, st, 0, bbytes);
        k_bwd_solve<TL, MULTI><<<std::min(grid, S.nbwd_items * ng), 256, sm, st>>>(
            D.fronts, S.bwd_items, S.nbwd_items, S.sync + 1, D.fv_pub_off + slots, D.fv_fronts, ab,
            S.gather_nch, S.gather_off, D.dinv_off, S.bwd_wlist, D.rows, Ls, Dinv, xp, fv, grp);
    }
}

template <typename TL>
void solve_levels(const DevPlan& D, const TL* Ls, const TL* Dinv, double* xp, double* fv, int nrhs,
                  cudaStream_t st) {
    if (nrhs == 1)
        solve_launch<TL, false>(D, Ls, Dinv, xp, fv, nrhs, st);
    else
        solve_launch<TL, true>(D, Ls, Dinv, xp, fv, nrhs, st);
}

template void solve_levels<double>(const DevPlan&, const double*, const double*, double*, double*,
                                   int, cudaStream_t);
template void solve_levels<float>(const DevPlan&, const float*, const float*, double*, double*, int,
                                  cudaStream_t);

}  // namespace mdgpu
