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

#include "device_common.cuh"
#include "kernels.hpp"

namespace mdgpu {

// Front vector of supernode s: rows fv_off[s] .. fv_off[s] + m - 1 of one
// array whose row holds the nrhs right-hand sides side by side, so row r,
// right-hand side q is front_vec(...)[r * nrhs + q].
template <typename TV>
__device__ inline TV* front_vec(TV* fv, const int64_t* fv_off, int s, int nrhs) {
    return fv + fv_off[s] * nrhs;
}

// ---------------------------------------------------------------------------
// one launch per level and direction: dependency-ordered tile tasks
//
// Each CTA takes the next task by an atomic ticket, so every task that
// started before it holds a lower ticket; the task lists are ordered so that
// a task only waits for tasks earlier in its list, hence for CTAs that are
// already resident, and the waits cannot deadlock.  A pivot tile publishes
// its solution values and then a flag (release); a dependent task polls the
// flag (acquire) with an iteration limit, after which the solve is aborted
// (every waiter leaves) and the error word is set for the host.
// ---------------------------------------------------------------------------

constexpr int kSolveWaitPolls = 1 << 18;  // ~0.1-0.3 s at ~1 us per poll
constexpr int kWarpSolveRhs = 4;   // right-hand sides per pass of the warp path
constexpr int kVecLD = kTile + 4;  // column stride of a vector block in shared memory: 4 mod 16
                                   // doubles, a conflict-free operand of the matrix instructions
constexpr int kGroupRhs = 8;       // right-hand sides of one group (a matrix instruction's columns)

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int ld_relaxed_gpu(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(int* p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// load of a value another CTA of this launch published (ordered after the
// acquire by the CTA barrier; never served from this SM's L1)
__device__ __forceinline__ double ld_shared_value(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

__device__ bool wait_flag(const int* flag, int target, int* abort_flag, int* err) {
    for (int it = 0; it < kSolveWaitPolls; ++it) {
        if (ld_acquire_gpu(flag) >= target) return true;
        if (ld_relaxed_gpu(abort_flag)) return false;
        __nanosleep(64);
    }
    atomicExch(abort_flag, 1);
    atomicOr(err, 1);
    return false;
}

// Published pivot-tile values: every slot starts as the all-ones bit pattern
// (a NaN that arithmetic never produces), and a producer stores final values
// only (aligned 8-byte stores are single-copy atomic), so a consumer that
// sees no sentinel has the data: one round trip instead of flag then data.
// All threads poll together (uniform result): the warps that hold slot
// elements spin on their own elements (a warp vote per round, no block
// barrier, a short sleep and an abort check every 32 rounds), the others go
// straight to the closing barrier; iteration limit as wait_flag.
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
// (src: the slot, column after column of 64 rows; dst: columns kVecLD apart)
__device__ bool poll_published(double* dst, const double* src, int nk, int nrhs, int* abort_flag,
                               int* err) {
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
                    atomicExch(abort_flag, 1);
                    atomicOr(err, 1);
                }
                ok = false;
                break;
            }
            if ((it & 31) == 31) {
                const int a = lane == 0 ? ld_relaxed_gpu(abort_flag) : 0;
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

template <typename TL>
__device__ __forceinline__ void cp_async_elem(TL* dst, const TL* src) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    if constexpr (sizeof(TL) == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
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
// large-front tile tasks: a pipeline of two stages streams the L blocks a
// task multiplies, each with the vector block it is multiplied by (a pivot
// tile's published solution, or gathered solution rows), by cp.async; the
// block in use is consumed while the next ones load.  Published vectors come
// through L2 (16-byte cp.async.cg); a stage whose copy still holds a
// sentinel falls back to polling that slot.
// ---------------------------------------------------------------------------

constexpr int kSolveStages = 2;

// shared memory of a tile task: the stages' L blocks, their vector blocks, a
// vector, the gather's row indices; one right-hand side also keeps the
// diagonal inverse in a block of its own (several take it through the stages,
// after the last L block)
template <typename TL, bool MULTI>
__host__ __device__ constexpr size_t level_smem_bytes() {
    return ((size_t)(kSolveStages + (MULTI ? 0 : 1)) * kTile * blk_ld<TL>()) * sizeof(TL) +
           (size_t)(kSolveStages + 1) * kVecLD * (MULTI ? kGroupRhs : 1) * sizeof(double) +
           (size_t)SolveScheduleHost::kGatherTiles * kTile * sizeof(int);
}

template <typename TL, bool MULTI>
struct LevelSmem {
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
        Dk = Lst + kSolveStages * T * LD;
        Vst = reinterpret_cast<double*>(Dk + (MULTI ? 0 : T * LD));
        Y = Vst + kSolveStages * VB;
        idx = reinterpret_cast<int*>(Y + VB);
    }
    __device__ TL* lb(int p) const { return Lst + (p % kSolveStages) * kTile * blk_ld<TL>(); }
    __device__ double* vb(int p) const { return Vst + (p % kSolveStages) * VB; }
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
                                            int* abort_flag, int* err) {
    bool mine = true;
    for (int e = threadIdx.x; e < kTile * nrhs; e += blockDim.x) {
        double& x = v[(e / kTile) * kVecLD + (e & (kTile - 1))];
        if ((e & (kTile - 1)) >= nk)
            x = 0.0;
        else if (is_unpublished(x))
            mine = false;
    }
    if (__syncthreads_and(mine)) return true;
    return poll_published(v, src, nk, nrhs, abort_flag, err);
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
                              double* __restrict__ pub, int* __restrict__ abort_flag,
                              int* __restrict__ err, const int64_t* __restrict__ fv_off,
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
    // this thread's row of tile i of the front vector
    auto gather_row = [&](int i) -> double {
        const TileRange ti = tile_range(i, F.m, F.c, T);
        const int R = ti.start + r;
        if (g != 0 || r >= ti.size) return 0.0;
        double x = R < F.c ? xp[F.first_col + R] : 0.0;
        const int e1 = amap_row[aoff + R + 1];
        for (int e = amap_row[aoff + R]; e < e1; ++e) x += __ldcg(fv + (int64_t)amap_ent[e]);
        return x;
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
    issue(0);
    double fcur = gather_row(i0), acc = 0.0;
    double fnext = cnt > 1 ? gather_row(i0 + 1) : 0.0;
    bool ok = true;
    for (int p = 0; p < P; ++p) {
        issue(p + 1);
        cp_async_wait_groups<1>();
        __syncthreads();
        const int i = i0 + p / kend, k = p % kend;
        double* Yk = sm.vb(p);
        if (!settle_slot(Yk, pb + (int64_t)k * T, min(T, F.c - k * T), 1, abort_flag, err)) {
            ok = false;
            break;
        }
        const TL* B = sm.lb(p);
#pragma unroll
        for (int l = 0; l < 16; ++l) acc += (double)B[db + r + (g + 4 * l) * LD] * Yk[g + 4 * l];
        if (!pivot && k == kend - 1) {  // update tile i complete: f_i - acc to the front vector
            const TileRange ti = tile_range(i, F.m, F.c, T);
            double v = acc + __shfl_xor_sync(0xffffffffu, acc, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            if (g == 0 && r < ti.size) f[ti.start + r] = fcur - v;
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
    const TL* Dk = sm.Dk;
    double a = acc + __shfl_xor_sync(0xffffffffu, acc, 8);
    a += __shfl_xor_sync(0xffffffffu, a, 16);
    if (g == 0) Y[r] = r < ti.size ? fcur - a : 0.0;
    __syncthreads();
    double y = 0.0;
#pragma unroll
    for (int l = 0; l < 16; ++l) y += (double)Dk[r + (g + 4 * l) * LD] * Y[g + 4 * l];
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
                               double* __restrict__ pub, int* __restrict__ abort_flag,
                               int* __restrict__ err, const int64_t* __restrict__ fv_off,
                               const int* __restrict__ amap_off, const int* __restrict__ amap_row,
                               const int* __restrict__ amap_ent,
                               const int64_t* __restrict__ dinv_off, const TL* __restrict__ Ls,
                               const TL* __restrict__ Dinv, double* __restrict__ xp,
                               double* __restrict__ fv, int n, int nrhs) {
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
        v[0] = v[1] = 0.0;
        if (r >= ti.size || !q0) return;
        if (R < F.c) {
            v[0] = xp[F.first_col + R + (int64_t)q * n];
            if (q1) v[1] = xp[F.first_col + R + (int64_t)(q + 1) * n];
        }
        const int e1 = amap_row[aoff + R + 1];
        for (int e = amap_row[aoff + R]; e < e1; ++e) {
            const double* w = fv + (int64_t)amap_ent[e] * nrhs + q;
            v[0] += __ldcg(w);
            if (q1) v[1] += __ldcg(w + 1);
        }
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
    issue(0);
    double fcur[2], fnext[2] = {0.0, 0.0}, acc[2][2] = {};
    gather_row(i0, fcur);
    if (cnt > 1) gather_row(i0 + 1, fnext);
    bool ok = true;
    for (int p = 0; p < P; ++p) {
        issue(p + 1);
        cp_async_wait_groups<1>();
        __syncthreads();
        const int i = i0 + p / kend, k = p % kend;
        if (!settle_slot(sm.vb(p), pb + (int64_t)k * T * nrhs, min(T, F.c - k * T), nrhs,
                         abort_flag, err)) {
            ok = false;
            break;
        }
        group_product<TL, false>(sm.lb(p), db, sm.vb(p), acc);
        if (!pivot && k == kend - 1) {  // update tile i complete
            const TileRange ti = tile_range(i, F.m, F.c, T);
            if (r < ti.size) {
                double* o = f + (int64_t)(ti.start + r) * nrhs + q;
                if (q0) o[0] = fcur[0] - (acc[0][0] + acc[1][0]);
                if (q1) o[1] = fcur[1] - (acc[0][1] + acc[1][1]);
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
            xp[F.first_col + ti.start + r + (int64_t)q * n] = y[0][0] + y[1][0];
            st_relaxed_f64(o + q * T, y[0][0] + y[1][0]);
        }
        if (q1) {
            xp[F.first_col + ti.start + r + (int64_t)(q + 1) * n] = y[0][1] + y[1][1];
            st_relaxed_f64(o + (q + 1) * T, y[0][1] + y[1][1]);
        }
    }
}

// Backward, update rows, task (s, j | h << 16): the partial sum
// L(k, j)' x_k over the update row tiles k of chunk h (kGatherTiles tiles;
// x final: ancestors, read through the row list) for pivot column tile j,
// written as a T x nrhs vector for the pivot task to add in chunk order, then
// counted in.  MULTI: a group of nrhs <= 8 right-hand sides on the matrix
// instructions; one: warp w takes columns 8w .. 8w + 7, lane (c1 = column,
// q1 = row phase) the rows q1, q1 + 4, ...: conflict-free reads of the stage
// layout, the phases summed by shuffles.
template <typename TL, bool MULTI>
__device__ void bwd_gather_task(int2 tk, const FrontDesc* __restrict__ fronts,
                                const int* __restrict__ rows, const int* __restrict__ gather_nch,
                                const int* __restrict__ gather_off, int* __restrict__ gcount,
                                const int64_t* __restrict__ dinv_off, const TL* __restrict__ Ls,
                                const double* __restrict__ xp, double* __restrict__ part, int n,
                                int nrhs) {
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
    __syncthreads();
    // two stages: the L blocks by cp.async; the ancestors' solution rows
    // (written in this launch) through L2 into registers one stage ahead,
    // stored into their stage after the previous stage's products
    constexpr int VPT = MULTI ? kTile * kGroupRhs / 256 : 1;
    double pend[VPT];
    auto fetch = [&](int p) {
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const int e = tid + 256 * k;
            pend[k] = 0.0;
            if (p < P && e < T * nrhs) {
                const int row = sm.idx[p * T + (e & (T - 1))], q = e / T;
                if (row >= 0) pend[k] = __ldcg(xp + row + (int64_t)q * n);
            }
        }
    };
    auto put = [&](int p) {
        if (p >= P) return;
        double* v = sm.vb(p);
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const int e = tid + 256 * k;
            if (e < T * nrhs) v[(e / T) * kVecLD + (e & (T - 1))] = pend[k];
        }
    };
    auto issue = [&](int p) {
        if (p < P) {
            const TileRange tkr = tile_range(k0 + p, F.m, F.c, T);
            load_block_async(sm.lb(p), Lc, F.ldl, tkr.start, tkr.size, tj.size);
        }
        cp_async_commit_group();
    };
    static_assert(kSolveStages == 2, "the gather's vector pipeline has two stages");
    issue(0);
    fetch(0);
    put(0);
    double acc[2][2] = {};
    for (int p = 0; p < P; ++p) {
        issue(p + 1);
        fetch(p + 1);
        cp_async_wait_groups<1>();
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
        if (q < nrhs) out[l + T * q] = acc[0][0] + acc[1][0];
        if (q + 1 < nrhs) out[l + T * (q + 1)] = acc[0][1] + acc[1][1];
    } else {
        double v = acc[0][0] + __shfl_xor_sync(0xffffffffu, acc[0][0], 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (q1 == 0) out[c1] = v;
    }
    // count this chunk in for the pivot task (s, j): the CTA's stores, then
    // a device-scope fence, then the increment
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        atomicAdd(gcount + dinv_off[s] / (T * T) + j, 1);
    }
}

// ---------------------------------------------------------------------------
// small fronts: a warp per front, the right-hand sides in passes of NQ
// (kWarpSolveRhs, or one), lane l holding rows l, l + 32, ... (R slots,
// m <= 32 R) of the pass's right-hand sides in registers.  Forward: the
// pivot value is broadcast by a shuffle and every lane updates its rows
// below it; backward: a warp reduction per pivot column (dot product with
// the final rows below it).  No block barriers; the children's update parts
// are summed into a per-warp shared buffer (child by child, deterministic)
// before the rows are taken into registers.
// ---------------------------------------------------------------------------

// Dependency words of the one-launch solve.  Forward: front s starts once
// done[s] (its finished children) reaches its child count, and counts
// itself in at its parent once its update rows are written.  Backward:
// front s starts once done[parent] reaches target[parent] (the parent's
// solution rows are final), and counts one completion of its own once its
// solution rows are written.  Data written inside the launch by other CTAs
// (children's update rows, ancestors' solution rows) are read through L2.
struct FrontDeps {
    int* done;
    const int* target;  // backward only
    int* abort_flag;
    int* err;
};

// Fronts of at most W rows (W = 8, 16, 32) on a group of W lanes of a warp
// (32 / W fronts per warp), one row per lane.  mask: the group's lanes; the
// group's rows of the warp buffer are wbuf[q * 32 + r].
template <int W>
__device__ __forceinline__ unsigned group_mask() {
    return W == 32 ? 0xffffffffu : (((1u << W) - 1u) << ((threadIdx.x & 31) & ~(W - 1)));
}

// the group's first lane waits (bounded) for *word >= target; uniform result
template <int W>
__device__ __forceinline__ bool group_wait(const int* word, int target, const FrontDeps& d,
                                           unsigned mask) {
    int ok = 1;
    if ((threadIdx.x & (W - 1)) == 0) ok = wait_flag(word, target, d.abort_flag, d.err) ? 1 : 0;
    return __shfl_sync(mask, ok, 0, W) != 0;
}
// every lane's stores, a device-scope fence, then one increment of *word
template <int W>
__device__ __forceinline__ void group_signal(int* word, unsigned mask) {
    __threadfence();
    __syncwarp(mask);
    if (word && (threadIdx.x & (W - 1)) == 0) atomicAdd(word, 1);
}

template <typename TL, typename TV, int W, int NQ>
__device__ void fwd_group_front(int s, const FrontDesc& F, const FrontDeps& deps,
                                const FrontDesc* __restrict__ fronts,
                                const int* __restrict__ child, const int* __restrict__ relmap,
                                const int64_t* __restrict__ fv_off, const TL* __restrict__ Ls,
                                TV* __restrict__ xp, TV* __restrict__ out, TV* __restrict__ fv,
                                int n, int nrhs, TV* wbuf) {
    const unsigned mask = group_mask<W>();
    if (!group_wait<W>(deps.done + s, F.child_end - F.child_beg, deps, mask)) return;
    const int r = threadIdx.x & (W - 1);
    const int m = F.m, c = F.c;
    const int64_t ldl = F.ldl;
    const TL* L = Ls + F.loff;
    for (int q0 = 0; q0 < nrhs; q0 += NQ) {
        const int nq = min(NQ, nrhs - q0);
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (q < nq && r < m)
                wbuf[q * 32 + r] = r < c ? xp[F.first_col + r + (int64_t)(q0 + q) * n] : TV(0);
        __syncwarp(mask);
        for (int h = F.child_beg; h < F.child_end; ++h) {  // children in order
            const int ch = child[h];
            const FrontDesc g = fronts[ch];
            const int uc = g.m - g.c;
            const TV* w = front_vec(fv, fv_off, ch, nrhs) + g.c * nrhs + q0;
            if (r < uc) {  // uc < m <= W
                const int p = relmap[g.rows_off + g.c + r];
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    if (q < nq) wbuf[q * 32 + p] += __ldcg(w + r * nrhs + q);
            }
            __syncwarp(mask);
        }
        TV v[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = (q < nq && r < m) ? wbuf[q * 32 + r] : TV(0);
        __syncwarp(mask);
        // column j of L for this lane's row, one column ahead of its use
        TV lc = (r > 0 && r < m) ? (TV)L[r] : TV(0), d = (TV)L[0];
        for (int j = 0; j < c; ++j) {
            TV ln = TV(0), dn = TV(1);
            if (j + 1 < c) {
                const TL* cn = L + (j + 1) * ldl;
                dn = (TV)cn[j + 1];
                ln = (r > j + 1 && r < m) ? (TV)cn[r] : TV(0);
            }
            // several right-hand sides: one reciprocal per column
            const TV rd = NQ > 1 ? TV(1) / d : TV(0);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const TV sv = __shfl_sync(mask, v[q], j, W);
                const TV y = NQ > 1 ? sv * rd : sv / d;
                if (r == j)
                    v[q] = y;
                else if (r > j)
                    v[q] -= lc * y;
            }
            lc = ln;
            d = dn;
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (q >= nq || r >= m) continue;
            if (r < c)
                xp[F.first_col + r + (int64_t)(q0 + q) * n] = v[q];
            else
                out[r * nrhs + q0 + q] = v[q];
        }
    }
    group_signal<W>(F.parent >= 0 ? deps.done + F.parent : nullptr, mask);
}

template <typename TL, typename TV, int W, int NQ>
__device__ void bwd_group_front(int s, const FrontDesc& F, const FrontDeps& deps,
                                const int* __restrict__ rows, const TL* __restrict__ Ls,
                                TV* __restrict__ xp, int n, int nrhs) {
    const unsigned mask = group_mask<W>();
    if (F.parent >= 0 && !group_wait<W>(deps.done + F.parent, deps.target[F.parent], deps, mask))
        return;
    const int r = threadIdx.x & (W - 1);
    const int m = F.m, c = F.c;
    const int64_t ldl = F.ldl;
    const TL* L = Ls + F.loff;
    // this lane's row in the solution: a pivot row, else an ancestor's
    const int src = r < c ? F.first_col + r : (r < m ? rows[F.rows_off + r] : 0);
    for (int q0 = 0; q0 < nrhs; q0 += NQ) {
        const int nq = min(NQ, nrhs - q0);
        TV v[NQ];  // y on the pivot rows (x once solved), final x on the others
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            v[q] = (q < nq && r < m) ? __ldcg(xp + src + (int64_t)(q0 + q) * n) : TV(0);
        const int jl = c - 1;
        TV lc = (r > jl && r < m) ? (TV)L[r + jl * ldl] : TV(0), d = (TV)L[jl + jl * ldl];
        for (int j = jl; j >= 0; --j) {
            TV ln = TV(0), dn = TV(1);
            if (j > 0) {
                const TL* cn = L + (j - 1) * ldl;
                dn = (TV)cn[j - 1];
                ln = (r > j - 1 && r < m) ? (TV)cn[r] : TV(0);
            }
            TV p[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q) p[q] = lc * v[q];
#pragma unroll
            for (int o = W / 2; o > 0; o >>= 1)
#pragma unroll
                for (int q = 0; q < NQ; ++q) p[q] += __shfl_xor_sync(mask, p[q], o, W);
            if (r == j) {
#pragma unroll
                for (int q = 0; q < NQ; ++q) v[q] = (v[q] - p[q]) / d;
            }
            lc = ln;
            d = dn;
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (q < nq && r < c) xp[F.first_col + r + (int64_t)(q0 + q) * n] = v[q];
    }
    group_signal<W>(deps.done + s, mask);
}

// Fronts of 33..160 rows: the same sweeps with the front vector kept in the
// warp's shared buffer (ld MR rows per right-hand side) instead of registers.
template <typename TL, typename TV, int NQ>
__device__ void fwd_warp_front_smem(int s, const FrontDesc& F, const FrontDeps& deps,
                                    const FrontDesc* __restrict__ fronts,
                                    const int* __restrict__ child, const int* __restrict__ relmap,
                                    const int64_t* __restrict__ fv_off, const TL* __restrict__ Ls,
                                    TV* __restrict__ xp, TV* __restrict__ out, TV* __restrict__ fv,
                                    int n, int nrhs, TV* f, int MR) {
    if (!group_wait<32>(deps.done + s, F.child_end - F.child_beg, deps, 0xffffffffu)) return;
    const int lane = threadIdx.x & 31;
    const int m = F.m, c = F.c;
    const int64_t ldl = F.ldl;
    const TL* L = Ls + F.loff;
    for (int q0 = 0; q0 < nrhs; q0 += NQ) {
        const int nq = min(NQ, nrhs - q0);
        for (int r = lane; r < m; r += 32)
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (q < nq)
                    f[q * MR + r] = r < c ? xp[F.first_col + r + (int64_t)(q0 + q) * n] : TV(0);
        __syncwarp();
        for (int h = F.child_beg; h < F.child_end; ++h) {  // children in order
            const int ch = child[h];
            const FrontDesc g = fronts[ch];
            const int uc = g.m - g.c;
            const TV* w = front_vec(fv, fv_off, ch, nrhs) + g.c * nrhs + q0;
            const int* rm = relmap + g.rows_off + g.c;
            for (int rr = lane; rr < uc; rr += 32) {
                const int p = rm[rr];
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    if (q < nq) f[q * MR + p] += __ldcg(w + rr * nrhs + q);
            }
            __syncwarp();
        }
        for (int j = 0; j < c; ++j) {
            const TL* col = L + j * ldl;
            const TV d = (TV)col[j];
            const TV rd = NQ > 1 ? TV(1) / d : TV(0);  // several right-hand sides
            TV y[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q) y[q] = NQ > 1 ? f[q * MR + j] * rd : f[q * MR + j] / d;
            if (lane == (j & 31)) {
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    if (q < nq) xp[F.first_col + j + (int64_t)(q0 + q) * n] = y[q];
            }
            for (int r = j + 1 + lane; r < m; r += 32) {
                const TV l = (TV)col[r];
#pragma unroll
                for (int q = 0; q < NQ; ++q) f[q * MR + r] -= l * y[q];
            }
            __syncwarp();
        }
        for (int r = c + lane; r < m; r += 32)
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (q < nq) out[r * nrhs + q0 + q] = f[q * MR + r];
        __syncwarp();
    }
    group_signal<32>(F.parent >= 0 ? deps.done + F.parent : nullptr, 0xffffffffu);
}

template <typename TL, typename TV, int NQ>
__device__ void bwd_warp_front_smem(int s, const FrontDesc& F, const FrontDeps& deps,
                                    const int* __restrict__ rows, const TL* __restrict__ Ls,
                                    TV* __restrict__ xp, int n, int nrhs, TV* x, int MR) {
    if (F.parent >= 0 &&
        !group_wait<32>(deps.done + F.parent, deps.target[F.parent], deps, 0xffffffffu))
        return;
    const int lane = threadIdx.x & 31;
    const int m = F.m, c = F.c;
    const int64_t ldl = F.ldl;
    const TL* L = Ls + F.loff;
    const int* rw = rows + F.rows_off;
    for (int q0 = 0; q0 < nrhs; q0 += NQ) {
        const int nq = min(NQ, nrhs - q0);
        for (int r = lane; r < m; r += 32) {
            const int src = r < c ? F.first_col + r : rw[r];
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                x[q * MR + r] = q < nq ? __ldcg(xp + src + (int64_t)(q0 + q) * n) : TV(0);
        }
        __syncwarp();
        for (int j = c - 1; j >= 0; --j) {
            const TL* col = L + j * ldl;
            TV p[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q) p[q] = TV(0);
            for (int r = j + 1 + lane; r < m; r += 32) {
                const TV l = (TV)col[r];
#pragma unroll
                for (int q = 0; q < NQ; ++q) p[q] += l * x[q * MR + r];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int q = 0; q < NQ; ++q) p[q] += __shfl_xor_sync(0xffffffffu, p[q], o);
            const TV d = (TV)col[j];
            if (lane == (j & 31)) {
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    const TV v = (x[q * MR + j] - p[q]) / d;
                    x[q * MR + j] = v;
                    if (q < nq) xp[F.first_col + j + (int64_t)(q0 + q) * n] = v;
                }
            }
            __syncwarp();
        }
    }
    group_signal<32>(deps.done + s, 0xffffffffu);
}

// dispatch on the front's rows: registers up to 32, the shared buffer above
template <typename TL, typename TV, int NQ>
__device__ void fwd_warp_front(int s, const FrontDeps& deps, const FrontDesc* __restrict__ fronts,
                               const int* __restrict__ child, const int* __restrict__ relmap,
                               const int64_t* __restrict__ fv_off, const TL* __restrict__ Ls,
                               TV* __restrict__ xp, TV* __restrict__ fv, int n, int nrhs,
                               TV* wbuf, int MR) {
    const FrontDesc F = fronts[s];
    TV* out = front_vec(fv, fv_off, s, nrhs);
    if (F.m <= 32)
        fwd_group_front<TL, TV, 32, NQ>(s, F, deps, fronts, child, relmap, fv_off, Ls, xp, out,
                                        fv, n, nrhs, wbuf);
    else
        fwd_warp_front_smem<TL, TV, NQ>(s, F, deps, fronts, child, relmap, fv_off, Ls, xp, out,
                                        fv, n, nrhs, wbuf, MR);
}

template <typename TL, typename TV, int NQ>
__device__ void bwd_warp_front(int s, const FrontDeps& deps, const FrontDesc* __restrict__ fronts,
                               const int* __restrict__ rows, const TL* __restrict__ Ls,
                               TV* __restrict__ xp, int n, int nrhs, TV* wbuf, int MR) {
    const FrontDesc F = fronts[s];
    if (F.m <= 32)
        bwd_group_front<TL, TV, 32, NQ>(s, F, deps, rows, Ls, xp, n, nrhs);
    else
        bwd_warp_front_smem<TL, TV, NQ>(s, F, deps, rows, Ls, xp, n, nrhs, wbuf, MR);
}

// per-warp shared buffer of the warp path: MR = rows rounded up to 32, times
// the right-hand sides of one pass
__host__ __device__ constexpr int warp_rows(int msmall) { return ((msmall + 31) / 32) * 32; }
__host__ __device__ constexpr int warp_buf_stride(int msmall, bool multi) {
    return warp_rows(msmall) * (multi ? kWarpSolveRhs : 1);
}

// Warp tasks of one warp item (its slice of the direction's warp list):
// tasks [0, n1) one front each, then two fronts of 9..16 rows per task, then
// four of at most 8 rows.
struct WarpTasks {
    const int* list;
    int n1, n2, n4;
    __host__ __device__ int count() const { return n1 + (n2 + 1) / 2 + (n4 + 3) / 4; }
};


template <typename TL, typename TV, int NQ>
__device__ void fwd_warp_task(const WarpTasks& wt, int t, const FrontDeps& deps,
                              const FrontDesc* __restrict__ fronts,
                              const int* __restrict__ child, const int* __restrict__ relmap,
                              const int64_t* __restrict__ fv_off, const TL* __restrict__ Ls,
                              TV* __restrict__ xp, TV* __restrict__ fv, int n, int nrhs, TV* wbuf,
                              int MR) {
    const int lane = threadIdx.x & 31;
    if (t < wt.n1) {
        fwd_warp_front<TL, TV, NQ>(wt.list[t], deps, fronts, child, relmap, fv_off, Ls, xp, fv, n,
                                   nrhs, wbuf, MR);
        return;
    }
    t -= wt.n1;
    const int t2 = (wt.n2 + 1) / 2;
    if (t < t2) {
        const int k = 2 * t + (lane >> 4);
        if (k < wt.n2) {
            const int s = wt.list[wt.n1 + k];
            const FrontDesc F = fronts[s];
            fwd_group_front<TL, TV, 16, NQ>(s, F, deps, fronts, child, relmap, fv_off, Ls, xp,
                                            front_vec(fv, fv_off, s, nrhs), fv, n, nrhs,
                                            wbuf + (lane & 16));
        }
        return;
    }
    const int k = 4 * (t - t2) + (lane >> 3);
    if (k < wt.n4) {
        const int s = wt.list[wt.n1 + wt.n2 + k];
        const FrontDesc F = fronts[s];
        fwd_group_front<TL, TV, 8, NQ>(s, F, deps, fronts, child, relmap, fv_off, Ls, xp,
                                       front_vec(fv, fv_off, s, nrhs), fv, n, nrhs,
                                       wbuf + (lane & 24));
    }
}

template <typename TL, typename TV, int NQ>
__device__ void bwd_warp_task(const WarpTasks& wt, int t, const FrontDeps& deps,
                              const FrontDesc* __restrict__ fronts, const int* __restrict__ rows,
                              const TL* __restrict__ Ls, TV* __restrict__ xp, int n, int nrhs,
                              TV* wbuf, int MR) {
    const int lane = threadIdx.x & 31;
    if (t < wt.n1) {
        bwd_warp_front<TL, TV, NQ>(wt.list[t], deps, fronts, rows, Ls, xp, n, nrhs, wbuf, MR);
        return;
    }
    t -= wt.n1;
    const int t2 = (wt.n2 + 1) / 2;
    if (t < t2) {
        const int k = 2 * t + (lane >> 4);
        if (k < wt.n2) {
            const int s = wt.list[wt.n1 + k];
            bwd_group_front<TL, TV, 16, NQ>(s, fronts[s], deps, rows, Ls, xp, n, nrhs);
        }
        return;
    }
    const int k = 4 * (t - t2) + (lane >> 3);
    if (k < wt.n4) {
        const int s = wt.list[wt.n1 + wt.n2 + k];
        bwd_group_front<TL, TV, 8, NQ>(s, fronts[s], deps, rows, Ls, xp, n, nrhs);
    }
}

// Backward, task (s, j): pivot column tile j of front s accumulates, once
// the update-row gathers of (s, j) have all counted in, their partial sums
// in chunk order, then acc += sum_{k > j} L(k, j)' x_k over the pivot tiles
// nt1-1 .. j+1 of this front as they publish, and solves
// x_j = inv(L_jj)' (y_j - acc).  MULTI as in bwd_gather_task.
template <typename TL, bool MULTI>
__device__ void bwd_chain_task(int2 tk, const FrontDesc* __restrict__ fronts,
                               double* __restrict__ pub, int* __restrict__ abort_flag,
                               int* __restrict__ err, const int* __restrict__ gather_nch,
                               const int* __restrict__ gather_off, const int* __restrict__ gcount,
                               const double* __restrict__ part,
                               const int64_t* __restrict__ dinv_off, const TL* __restrict__ Ls,
                               const TL* __restrict__ Dinv, double* __restrict__ xp, int n,
                               int nrhs) {
    constexpr int T = kTile, LD = blk_ld<TL>();
    const LevelSmem<TL, MULTI> sm;
    __shared__ int s_ok;
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
    issue(0);
    double acc[2][2] = {};
    // this tile's y_j, before the first wait
    const int64_t xj = F.first_col + tj.start + l;
    const bool in = l < tj.size;
    const double y0 = in && own0 ? __ldcg(xp + xj + (int64_t)q * n) : 0.0;
    const double y1 = in && own1 ? __ldcg(xp + xj + (int64_t)(q + 1) * n) : 0.0;
    // the update-row partial sums of (s, j) (gathers hold lower tickets), in
    // chunk order, before the chain's first wait
    {
        const int nch = gather_nch[s];
        if (nch > 0) {
            if (tid == 0) s_ok = wait_flag(gcount + tile0 + j, nch, abort_flag, err) ? 1 : 0;
            __syncthreads();
            if (!s_ok) {
                cp_async_wait_groups<0>();
                return;
            }
            const double* pj = part + ((int64_t)gather_off[s] + (int64_t)j * nch) * T * nrhs;
            for (int h = 0; h < nch; ++h, pj += (int64_t)T * nrhs) {
                if (own0) acc[0][0] += __ldcg(pj + l + T * q);
                if (own1) acc[0][1] += __ldcg(pj + l + T * (q + 1));
            }
        }
    }
    bool ok = true;
    for (int p = 0; p < P; ++p) {
        issue(p + 1);
        cp_async_wait_groups<1>();
        __syncthreads();
        const int k = nt1 - 1 - p;
        double* X = sm.vb(p);
        if (!settle_slot(X, pb + (int64_t)k * T * nrhs, tile_range(k, F.m, F.c, T).size, nrhs,
                         abort_flag, err)) {
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
            xp[xj + (int64_t)q * n] = x[0][0] + x[1][0];
            st_relaxed_f64(pb + ((int64_t)j * nrhs + q) * T + l, x[0][0] + x[1][0]);
        }
        if (in && own1) {
            xp[xj + (int64_t)(q + 1) * n] = x[0][1] + x[1][1];
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
            xp[xj] = x;
            st_relaxed_f64(pb + (int64_t)j * T + l, x);
        }
    }
}

// ---------------------------------------------------------------------------
// forward update tiles with one right-hand side: L read straight from global
// memory into registers, coalesced (a thread per row), the next columns'
// loads issued before the current ones are used, no block barrier per L
// block.  The pivot tiles' published vectors come through poll_published
// into a shared double buffer (a buffer is rewritten two polls later, after
// the barrier of the poll between).
// ---------------------------------------------------------------------------

// (fronts of one pivot tile only: with more, one column group of loads in
// flight per iteration leaves a tail of one memory latency per 16 columns
// after the last pivot tile, where the staged tile path keeps two 64-column
// blocks in flight)
constexpr int kRt1MaxPivotTiles = 1;

struct Rt1Smem {
    double* Ys;  // 2 x T: published slots
    __device__ Rt1Smem() {
        extern __shared__ __align__(16) unsigned char smem_raw[];
        Ys = reinterpret_cast<double*>(smem_raw);
    }
};
template <typename TL>
__host__ __device__ constexpr size_t rt1_smem_bytes() {
    return 2 * (size_t)kTile * sizeof(double);
}

template <typename TL>
__device__ __forceinline__ TL ldL(const TL* p) {
    return __ldg(p);
}

// Forward update rows [R0, R1) of front s (at most 256; one right-hand side):
// thread = row; columns in groups of 16, the next group's loads issued
// before the current group's products.
template <typename TL>
__device__ void fwd_update_rt1(int s, int R0, int R1, const FrontDesc& F, double* __restrict__ pb,
                               int* __restrict__ abort_flag, int* __restrict__ err,
                               const int* __restrict__ amap_off, const int* __restrict__ amap_row,
                               const int* __restrict__ amap_ent, const TL* __restrict__ Ls,
                               const double* __restrict__ xp, double* __restrict__ f,
                               const double* __restrict__ fv) {
    constexpr int T = kTile;
    const Rt1Smem sm;
    const int R = R0 + threadIdx.x;
    const bool rv = R < R1;
    const TL* Lr = Ls + F.loff + R;
    double f0 = 0.0;
    if (rv) {
        const int* ar = amap_row + amap_off[s] + R;
        const int e0 = ar[0], e1 = ar[1];
        for (int e = e0; e < e1; ++e) f0 += __ldcg(fv + amap_ent[e]);
    }
    constexpr int GW = sizeof(TL) == 4 ? 16 : 8;  // columns per group (registers)
    constexpr int GPB = T / GW;                     // groups per 64-column block
    const int ng = (F.c + GW - 1) / GW;
    auto load = [&](int cg, TL (&v)[GW]) {
#pragma unroll
        for (int l = 0; l < GW; ++l) {
            const int col = GW * cg + l;
            v[l] = (rv && col < F.c) ? ldL(Lr + (int64_t)col * F.ldl) : TL(0);
        }
    };
    double acc = 0.0;
    TL lv[GW], ln[GW];
    load(0, lv);
    for (int cg = 0; cg < ng; ++cg) {
        if (cg + 1 < ng) load(cg + 1, ln);
        const int k = cg / GPB;
        double* Yk = sm.Ys + (k & 1) * T;
        if (cg % GPB == 0 &&
            !poll_published(Yk, pb + (int64_t)k * T, min(T, F.c - k * T), 1, abort_flag, err))
            return;
        const double* y = Yk + GW * (cg % GPB);
#pragma unroll
        for (int l = 0; l < GW; ++l) acc += (double)lv[l] * y[l];
#pragma unroll
        for (int l = 0; l < GW; ++l) lv[l] = ln[l];
    }
    if (rv) f[R] = f0 - acc;
}

// One launch per direction over all work items (the item lists, in a
// topological order by critical-path priority, and their kinds are
// described with the solve schedule): persistent CTAs take items by atomic
// ticket.  An item only waits for items with lower tickets -- children's
// (forward) and parents' (backward) items come earlier in the list, and so
// do a front's earlier pivot tiles and its backward gathers -- and a CTA
// takes a ticket only while it runs, so every wait is for a CTA that is
// running or done.
// Forward: a front's items wait for its children (the count of finished
// children), a small front counts itself in at its parent once written, a
// large front once its last update tile is (a per-front count of finished
// update tiles).  Backward: a front's items wait for its parent's solution
// rows (the parent's count of completions: one per pivot tile of a large
// front, one for a small front); the pivot tasks wait for their gathers'
// counts as before.  Every wait polls with an iteration limit; on timeout
// the launch is aborted (every later wait returns at once) and the error
// word reaches the host.

// a CTA's tid 0 waits (bounded) for *word >= target; uniform result
__device__ __forceinline__ bool cta_wait(const int* word, int target, int* abort_flag, int* err) {
    __shared__ int s_wok;
    if (threadIdx.x == 0) s_wok = wait_flag(word, target, abort_flag, err) ? 1 : 0;
    __syncthreads();
    return s_wok != 0;
}

// A group's own words in the sync array (its front counts and gather counts)
// and its slices of the work vectors.
struct SolveGroups {
    int n, nrhs;        // unknowns, right-hand sides of the launch
    int stride;         // sync words of a group
    int64_t fv_total;   // work vector rows
    __device__ int count() const { return (nrhs + kGroupRhs - 1) / kGroupRhs; }
    __device__ int size(int g) const { return min(kGroupRhs, nrhs - kGroupRhs * g); }
    __device__ int64_t xp_off(int g) const { return (int64_t)kGroupRhs * g * n; }
    __device__ int64_t fv_off(int g) const { return kGroupRhs * fv_total * g; }
};

// residency by shared memory: one right-hand side keeps three blocks of L per
// CTA (FP32 52 KB, FP64 104 KB), a group two and its vectors (49 and 83 KB)
template <typename TL, bool MULTI>
constexpr int solve_ctas_per_sm() {
    return sizeof(TL) == 8 ? 2 : MULTI ? 3 : 4;
}

template <typename TL, bool MULTI>
__global__ void __launch_bounds__(256, solve_ctas_per_sm<TL, MULTI>())
    k_fwd_solve(const FrontDesc* __restrict__ fronts, const int4* __restrict__ items, int nitems,
                int* __restrict__ counter, int64_t pub_rows, int* __restrict__ abort_flag,
                int* __restrict__ err, int* __restrict__ fdone0, int* __restrict__ udone0,
                const int64_t* __restrict__ fv_off, const int* __restrict__ amap_off,
                const int* __restrict__ amap_row, const int* __restrict__ amap_ent,
                const int64_t* __restrict__ dinv_off, const int* __restrict__ wlist,
                const int* __restrict__ child,
                const int* __restrict__ relmap, const TL* __restrict__ Ls,
                const TL* __restrict__ Dinv, double* __restrict__ xp0, double* __restrict__ fv0,
                SolveGroups grp, int MR) {
    constexpr int T = kTile;
    __shared__ int s_item;
    const int ngroups = MULTI ? grp.count() : 1, n = grp.n;
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
        int* fdone = fdone0 + gi * grp.stride;
        int* udone = udone0 + gi * grp.stride;
        const FrontDeps deps{fdone, nullptr, abort_flag, err};
        if (it.x == SolveScheduleHost::kItemWarps) {
            extern __shared__ __align__(16) unsigned char smem_raw[];
            const WarpTasks wt{wlist + it.y, it.z & 0xff, (it.z >> 8) & 0xff, it.z >> 16};
            const int w = threadIdx.x >> 5, t = w;
            double* wbuf = reinterpret_cast<double*>(smem_raw) + w * warp_buf_stride(MR, MULTI);
            if (t < wt.count())
                fwd_warp_task<TL, double, MULTI ? kWarpSolveRhs : 1>(
                    wt, t, deps, fronts, child, relmap, fv_off, Ls, xp, fv, n, nrhs, wbuf, MR);
        } else {
            // a tile task of a large front: its children first
            const int2 tk = make_int2(it.y, it.z);
            const int s = tk.x, i0 = tk.y & 0xffff, cnt = tk.y >> 16;
            const FrontDesc F = fronts[s];
            const int nt1 = tiles_l(F.c, T);
            if (cta_wait(fdone + s, F.child_end - F.child_beg, abort_flag, err)) {
                if constexpr (MULTI) {
                    fwd_tile_group<TL>(tk, fronts, pub, abort_flag, err, fv_off, amap_off,
                                       amap_row, amap_ent, dinv_off, Ls, Dinv, xp, fv, n, nrhs);
                } else if (i0 >= nt1 && nt1 <= kRt1MaxPivotTiles) {
                    // update tiles of fronts with at most kRt1MaxPivotTiles
                    // pivot tiles, one right-hand side: registers straight
                    // from L (measured faster there; the staged pipeline
                    // streams long column ranges better)
                    double* pb = pub + (dinv_off[s] / (T * T)) * T;
                    const TileRange a = tile_range(i0, F.m, F.c, T);
                    const TileRange b = tile_range(i0 + cnt - 1, F.m, F.c, T);
                    fwd_update_rt1<TL>(s, a.start, b.start + b.size, F, pb, abort_flag, err,
                                       amap_off, amap_row, amap_ent, Ls, xp,
                                       front_vec(fv, fv_off, s, 1), fv);
                } else {
                    fwd_tile_task<TL>(tk, fronts, pub, abort_flag, err, fv_off, amap_off,
                                      amap_row, amap_ent, dinv_off, Ls, Dinv, xp, fv);
                }
                // update tiles counted in; the front's last one counts the
                // front in at its parent
                if (i0 >= nt1) {
                    __syncthreads();
                    if (threadIdx.x == 0) {
                        __threadfence();
                        const int ntu = tiles_l(F.m - F.c, T);
                        if (atomicAdd(udone + s, cnt) + cnt == ntu && F.parent >= 0) {
                            __threadfence();
                            atomicAdd(fdone + F.parent, 1);
                        }
                    }
                }
            }
        }
        __syncthreads();  // shared memory and s_item free for the next item
    }
}

template <typename TL, bool MULTI>
__global__ void __launch_bounds__(256, solve_ctas_per_sm<TL, MULTI>())
    k_bwd_solve(const FrontDesc* __restrict__ fronts, const int4* __restrict__ items, int nitems,
                int* __restrict__ counter, int64_t pub_rows, int64_t part_rows,
                int* __restrict__ abort_flag, int* __restrict__ err, int* __restrict__ bdone0,
                const int* __restrict__ btarget, const int* __restrict__ gather_nch,
                const int* __restrict__ gather_off, int* __restrict__ gcount0,
                const int64_t* __restrict__ dinv_off, const int* __restrict__ wlist,
                const int* __restrict__ rows, const TL* __restrict__ Ls,
                const TL* __restrict__ Dinv, double* __restrict__ xp0, double* __restrict__ fv0,
                SolveGroups grp, int MR) {
    __shared__ int s_item;
    const int ngroups = MULTI ? grp.count() : 1, n = grp.n;
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
        double* part = fv + part_rows * nrhs;
        int* bdone = bdone0 + gi * grp.stride;
        int* gcount = gcount0 + gi * grp.stride;
        const FrontDeps deps{bdone, btarget, abort_flag, err};
        if (it.x == SolveScheduleHost::kItemWarps) {
            extern __shared__ __align__(16) unsigned char smem_raw[];
            const WarpTasks wt{wlist + it.y, it.z & 0xff, (it.z >> 8) & 0xff, it.z >> 16};
            const int w = threadIdx.x >> 5, t = w;
            double* wbuf = reinterpret_cast<double*>(smem_raw) + w * warp_buf_stride(MR, MULTI);
            if (t < wt.count())
                bwd_warp_task<TL, double, MULTI ? kWarpSolveRhs : 1>(wt, t, deps, fronts, rows, Ls,
                                                                     xp, n, nrhs, wbuf, MR);
        } else if (it.x == SolveScheduleHost::kItemGather) {
            // the update rows' partial sums need the ancestors' solution
            const int2 tk = make_int2(it.y, it.z);
            const int p = fronts[tk.x].parent;
            if (p < 0 || cta_wait(bdone + p, btarget[p], abort_flag, err))
                bwd_gather_task<TL, MULTI>(tk, fronts, rows, gather_nch, gather_off, gcount,
                                           dinv_off, Ls, xp, part, n, nrhs);
        } else {
            // a pivot tile: its gathers (counted) waited for the ancestors
            const int2 tk = make_int2(it.y, it.z);
            bwd_chain_task<TL, MULTI>(tk, fronts, pub, abort_flag, err, gather_nch, gather_off,
                                      gcount, part, dinv_off, Ls, Dinv, xp, n, nrhs);
            __syncthreads();
            if (threadIdx.x == 0) {
                __threadfence();
                atomicAdd(bdone + tk.x, 1);
            }
        }
        __syncthreads();  // shared memory and s_item free for the next item
    }
}

// Before the sweeps: the sync words cleared, every group's publication slots
// set to the unpublished pattern.
__global__ void __launch_bounds__(256)
    k_solve_init(int4* __restrict__ sync, int64_t nsync4, double* __restrict__ fv0,
                 int64_t pub_rows, int64_t slot_rows, SolveGroups grp) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = tid; i < nsync4; i += nt) sync[i] = make_int4(0, 0, 0, 0);
    for (int g = 0; g < grp.count(); ++g) {
        // slots start on 16 bytes and hold 64 rows each
        double2* p = reinterpret_cast<double2*>(fv0 + grp.fv_off(g) + pub_rows * grp.size(g));
        const int64_t cnt = slot_rows * grp.size(g) / 2;
        const double v = __longlong_as_double(-1ll);
        for (int64_t i = tid; i < cnt; i += nt) p[i] = make_double2(v, v);
    }
}

// ---------------------------------------------------------------------------
// permutations
// ---------------------------------------------------------------------------

__global__ void k_perm_gather(const int* __restrict__ perm, const double* __restrict__ b,
                              double* __restrict__ xp, int n, int nrhs, int ldb) {
    int64_t total = (int64_t)n * nrhs;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int q = (int)(idx / n), k = (int)(idx - (int64_t)q * n);
        xp[idx] = b[(perm ? perm[k] : k) + (int64_t)q * ldb];
    }
}

__global__ void k_perm_scatter(const int* __restrict__ perm, const double* __restrict__ xp,
                               double* __restrict__ x, int n, int nrhs, int ldx) {
    int64_t total = (int64_t)n * nrhs;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int q = (int)(idx / n), k = (int)(idx - (int64_t)q * n);
        x[(perm ? perm[k] : k) + (int64_t)q * ldx] = xp[idx];
    }
}

void permute_gather(const int* perm, const double* b, double* xp, int n, int nrhs, int ldb,
                    cudaStream_t st) {
    int64_t total = (int64_t)n * nrhs;
    int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 16);
    k_perm_gather<<<blocks, 256, 0, st>>>(perm, b, xp, n, nrhs, ldb);
}

void permute_scatter(const int* perm, const double* xp, double* x, int n, int nrhs, int ldx,
                     cudaStream_t st) {
    int64_t total = (int64_t)n * nrhs;
    int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 16);
    k_perm_scatter<<<blocks, 256, 0, st>>>(perm, xp, x, n, nrhs, ldx);
}

// ---------------------------------------------------------------------------
// launch sequence
// ---------------------------------------------------------------------------

// rows of a small front's warp buffer (every level's largest small front)
constexpr int kWarpBufRows = ((Plan::kSmallMaxRows + 31) / 32) * 32;

// dynamic shared memory of a solve launch: the tile tasks' stages or the
// eight warps' buffers, whichever is larger
template <typename TL, bool MULTI>
static size_t solve_smem() {
    size_t m = level_smem_bytes<TL, MULTI>();
    if (!MULTI) m = std::max(m, rt1_smem_bytes<TL>());
    return std::max(m, 8 * (size_t)warp_buf_stride(kWarpBufRows, MULTI) * sizeof(double));
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

int solve_groups(int nrhs) { return nrhs == 1 ? 1 : (nrhs + kGroupRhs - 1) / kGroupRhs; }
int64_t solve_sync_words(int nflags, int nfronts, int groups) {
    return (4 + (int64_t)groups * (nflags + 3 * (int64_t)nfronts) + 3) & ~(int64_t)3;
}

template <typename TL, bool MULTI>
static void solve_launch(const DevPlan& D, const TL* Ls, const TL* Dinv, double* xp, double* fv,
                         int nrhs, cudaStream_t st) {
    const SolveSchedule& S = D.solve;
    static_assert(Plan::kSmallMaxRows <= 32 * 5, "the warp path holds 160 rows in shared memory");
    // sync: the two ticket counters and the abort word, then per group the
    // gathers' counts per pivot tile, and per front the forward
    // finished-children and finished-update-tile counts and the backward
    // completions
    int* counters = S.sync;
    int* abort_flag = S.sync + 2;
    int* gcount = S.sync + 4;
    int* fdone = gcount + S.nflags;
    int* udone = fdone + S.nfronts;
    int* bdone = udone + S.nfronts;
    const SolveGroups grp{D.n, nrhs, S.nflags + 3 * S.nfronts, D.fv_total};
    const int64_t slots = (int64_t)S.nflags * kTile;  // rows of one direction
    const int64_t nsync = solve_sync_words(S.nflags, S.nfronts, solve_groups(nrhs));
    const int sms = D.num_sms > 0 ? D.num_sms : 148;
    {
        const int64_t work = std::max(nsync / 4, slots * nrhs);
        const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((work + 1023) / 1024, sms * 8));
        k_solve_init<<<blocks, 256, 0, st>>>(reinterpret_cast<int4*>(S.sync), nsync / 4, fv,
                                             D.fv_pub_off, 2 * slots, grp);
    }
    const size_t sm = solve_smem<TL, MULTI>();
    const int grid = sms * solve_ctas_per_sm<TL, MULTI>();
    const int ng = MULTI ? solve_groups(nrhs) : 1;
    double fbytes = 0, bbytes = 0;
    for (int l = 0; l < D.nlevels; ++l) {
        fbytes += (S.small_elems[l] + S.fwd_elems[l]) * sizeof(TL);
        bbytes += (S.small_elems[l] + S.bwd_elems[l]) * sizeof(TL);
    }
    if (S.nfwd_items > 0) {
        ProfScope ps(D.prof, KC_SOLVE_LARGE, st, 0, fbytes);
        k_fwd_solve<TL, MULTI><<<std::min(grid, S.nfwd_items * ng), 256, sm, st>>>(
            D.fronts, S.fwd_items, S.nfwd_items, counters, D.fv_pub_off, abort_flag,
            S.err, fdone, udone, D.fv_off, S.amap_off, S.amap_row, S.amap_ent, D.dinv_off,
            S.fwd_wlist, D.child, D.relmap, Ls, Dinv, xp, fv, grp, kWarpBufRows);
    }
    if (S.nbwd_items > 0) {
        ProfScope ps(D.prof, KC_SOLVE_LARGE, st, 0, bbytes);
        k_bwd_solve<TL, MULTI><<<std::min(grid, S.nbwd_items * ng), 256, sm, st>>>(
            D.fronts, S.bwd_items, S.nbwd_items, counters + 1, D.fv_pub_off + slots, D.fv_fronts,
            abort_flag, S.err, bdone, S.bwd_target, S.gather_nch, S.gather_off, gcount,
            D.dinv_off, S.bwd_wlist, D.rows, Ls, Dinv, xp, fv, grp, kWarpBufRows);
    }
}

template <typename TL, typename TV>
void solve_levels(const DevPlan& D, const TL* Ls, const TL* Dinv, TV* xp, TV* fv, int nrhs,
                  cudaStream_t st) {
    // as many groups of right-hand sides per launch as the sync words hold
    // (the work vectors are reused by the next launch)
    const int pass = kGroupRhs * D.solve.sync_groups;
    for (int q0 = 0; q0 < nrhs; q0 += pass) {
        const int nq = std::min(pass, nrhs - q0);
        double* x = xp + (int64_t)q0 * D.n;
        if (nq == 1)
            solve_launch<TL, false>(D, Ls, Dinv, x, fv, nq, st);
        else
            solve_launch<TL, true>(D, Ls, Dinv, x, fv, nq, st);
    }
}

template void solve_levels<double, double>(const DevPlan&, const double*, const double*, double*,
                                           double*, int, cudaStream_t);
template void solve_levels<float, double>(const DevPlan&, const float*, const float*, double*,
                                          double*, int, cudaStream_t);

}  // namespace mdgpu
