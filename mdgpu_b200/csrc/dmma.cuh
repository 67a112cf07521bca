// FP64 tensor-core products: mma.sync m16n8k16 (FP64 has no tcgen05 kind, so
// the warp-level instruction is the FP64 matrix path of sm_100a; measured on
// B200, 4 warps per SM of independent chains: 35.4 TFLOP/s against 28.2 for
// register FMAs, one instruction issued per 2048 multiply-adds).
//
// A warp's operand blocks sit in shared memory K-slowest: element (row, k) at
// [k * LD + row], LD = 4 mod 16 doubles.  The instruction's row g pairs with
// row 2 g of a 16-row block and row g + 8 with row 2 g + 1 (any bijection
// works as long as the accumulator is read back the same way), so both come
// from one 16-byte load, and LD = 4 mod 16 spreads the four k of a quarter
// warp over all banks.  Columns likewise: of a 16-column block the even
// columns form one 8-column operand and the odd ones the next.
#pragma once

#include <cuda_runtime.h>

namespace mdgpu {

__device__ __forceinline__ void dmma_16816(double (&c)[4], const double (&a)[8],
                                           const double (&b)[4]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3},"
        "{%4,%5,%6,%7,%8,%9,%10,%11},{%12,%13,%14,%15},{%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]),
          "d"(b[0]), "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

// acc += A B' over 16 steps of k: A 16 MT rows from As, B 16 NT rows from Bs
// (both at this warp's first row).  Accumulator (m, n, h, e) is row 16 m +
// 2 g + (e >> 1), column 16 n + 4 t + 2 (e & 1) + h, g = lane / 4, t =
// lane % 4: a lane's four columns 4 t .. 4 t + 3 of two adjacent rows.
template <int MT, int NT, int LDA, int LDB>
__device__ __forceinline__ void dmma_k16(const double* As, const double* Bs,
                                         double (&acc)[MT][NT][2][4]) {
    static_assert(LDA % 16 == 4 && LDB % 16 == 4, "bank spread of the four k of a quarter warp");
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    double a[MT][8];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double2 v =
                *reinterpret_cast<const double2*>(As + (4 * q + t) * LDA + 16 * m + 2 * g);
            a[m][2 * q] = v.x;
            a[m][2 * q + 1] = v.y;
        }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        double b[2][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double2 v =
                *reinterpret_cast<const double2*>(Bs + (4 * q + t) * LDB + 16 * n + 2 * g);
            b[0][q] = v.x;
            b[1][q] = v.y;
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h) dmma_16816(acc[m][n][h], a[m], b[h]);
    }
}

}  // namespace mdgpu
