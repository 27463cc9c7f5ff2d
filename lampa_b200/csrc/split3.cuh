// fp32 operands on the tensor cores: a float as the sum of three bf16 pieces (8 significant bits each).  Of the nine products of
// two such sums the six larger ones are issued, smallest first; the other three are below 2^-24 of the result.
#pragma once
#include "common.cuh"

namespace lampa {

struct Split3 { uint32_t h, m, l; };
__device__ __forceinline__ Split3 split3(float x, float y) {
    Split3 s;
    s.h = pack_bf16x2(x, y);
    const float2 h = unpack_bf16x2(s.h);
    const float rx = x - h.x, ry = y - h.y;
    s.m = pack_bf16x2(rx, ry);
    const float2 m = unpack_bf16x2(s.m);
    s.l = pack_bf16x2(rx - m.x, ry - m.y);
    return s;
}

// c[x] (16 x 8 n_tiles at row m0, column n0) += A[x] B over k in [k0, k1), a multiple of 16 long, for NA left operands with the same right
// one.  All are fp32 tiles in shared memory: A[m][k] (A_T: A[k][m]), B[k][n] (B_T: B[n][k]).  Only the rows k in [b0, b1) of B count.
template <int NA, int NT, bool A_T, bool B_T>
__device__ __forceinline__ void tile_product3(float (&c)[NA][NT][4], const float* const (&A)[NA], int lda, int m0, const float* B, int ldb,
                                              int n0, int n_tiles, int k0, int k1, int lane, int b0 = 0, int b1 = 1 << 20) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll 1
    for (int k = k0; k < k1; k += 16) {
        uint32_t a[NA][3][4];
#pragma unroll
        for (int x = 0; x < NA; ++x)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int m = m0 + g + 8 * (q & 1), kk = k + 2 * t + 8 * (q >> 1);
                const float2 v = A_T ? make_float2(A[x][kk * lda + m], A[x][(kk + 1) * lda + m]) : *reinterpret_cast<const float2*>(A[x] + m * lda + kk);
                const Split3 s = split3(v.x, v.y);
                a[x][0][q] = s.h; a[x][1][q] = s.m; a[x][2][q] = s.l;
            }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            if (nt >= n_tiles) break;
            uint32_t b[3][2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int n = n0 + 8 * nt + g, kk = k + 2 * t + 8 * q;
                float2 v = B_T ? *reinterpret_cast<const float2*>(B + n * ldb + kk) : make_float2(B[kk * ldb + n], B[(kk + 1) * ldb + n]);
                if (kk < b0 || kk >= b1) v.x = 0.f;
                if (kk + 1 < b0 || kk + 1 >= b1) v.y = 0.f;
                const Split3 s = split3(v.x, v.y);
                b[0][q] = s.h; b[1][q] = s.m; b[2][q] = s.l;
            }
#pragma unroll
            for (int x = 0; x < NA; ++x) {
                mma16816(c[x][nt], a[x][2], b[0][0], b[0][1]);
                mma16816(c[x][nt], a[x][0], b[2][0], b[2][1]);
                mma16816(c[x][nt], a[x][1], b[1][0], b[1][1]);
                mma16816(c[x][nt], a[x][1], b[0][0], b[0][1]);
                mma16816(c[x][nt], a[x][0], b[1][0], b[1][1]);
                mma16816(c[x][nt], a[x][0], b[0][0], b[0][1]);
            }
        }
    }
}

}  // namespace lampa
