// FP64 products of one output tile per CTA (sm_100a).
//
// A task kernel gives each CTA one TS x TS tile of a product and adds as many
// terms into its accumulators as the tile needs before it is written once.  The
// K slabs (32 deep) come through a three-stage cp.async pipeline with one
// barrier per slab; operands are laid out in shared memory as in global memory
// (K-contiguous operands [row][k], the others [k][row]), both with a row stride
// of 4 mod 16 doubles: copies and m8n8k4 fragment loads are free of bank
// conflicts.  TS = 64: 8 warps of 32 x 16; TS = 32 and 16: 4 warps of 16 x 16
// and 8 x 8, so that small knot counts do not multiply padding.
#pragma once

#include "mra_device.cuh"

namespace mra {

template <int TS>
struct Tile {
    static constexpr int NT = TS == 64 ? 256 : 128;    // threads of the CTA
    static constexpr int CTAS = TS == 64 ? 2 : 4;      // per SM (shared memory: 111, 55 or 28 KB each)
    static constexpr int WM = 2, WN = NT / 64;         // warps along rows / columns
    static constexpr int MI = TS / WM / 8, NJ = TS / WN / 8;
    static constexpr int RS = TS + 4;
    static constexpr int SLAB = TS * KS64 > TK64 * RS ? TS * KS64 : TK64 * RS;
    struct Smem {
        double A[3][SLAB];
        double B[3][SLAB];
    };
    struct Acc {
        double v[MI][NJ][2];
    };

    static __device__ __forceinline__ void zero(Acc& c) {
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) c.v[i][j][0] = c.v[i][j][1] = 0.0;
    }
    // row / column of accumulator (i, j, h) of this thread
    static __device__ __forceinline__ int row(int i) {
        const int w = threadIdx.x >> 5;
        return (w % WM) * (8 * MI) + 8 * i + ((threadIdx.x & 31) >> 2);
    }
    static __device__ __forceinline__ int col(int j, int h) {
        const int w = threadIdx.x >> 5;
        return (w / WM) * (8 * NJ) + 8 * j + 2 * (threadIdx.x & 3) + h;
    }
    // c += s * C (C: M x N, column-major)
    static __device__ __forceinline__ void add(Acc& c, double s, const double* C, long ldc, int M, int N) {
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = row(i), q = col(j, h);
                    if (r < M && q < N) c.v[i][j][h] += s * C[r + (long)q * ldc];
                }
    }
    // C = s * c
    static __device__ __forceinline__ void store(const Acc& c, double s, double* C, long ldc, int M, int N) {
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = row(i), q = col(j, h);
                    if (r < M && q < N) C[r + (long)q * ldc] = s * c.v[i][j][h];
                }
    }

    // One slab of an operand: R valid rows (of TS), rows KC-contiguous ([row][k]:
    // element (i, k) at X[k + i ld]) or row-contiguous (X[i + k ld]); zeros beyond
    // the valid rows and K.  vec: pairs by 16-byte copies (X 16-byte aligned, ld
    // even, and R (row-contiguous) or K (K-contiguous) even).
    template <bool KC>
    static __device__ __forceinline__ void stage(double* s, const double* X, long ld, int R, int k0, int K, bool vec) {
        const int tid = threadIdx.x;
        if (vec) {
#pragma unroll
            for (int q = 0; q < TS * (TK64 / 2) / NT; ++q) {
                const int e = tid + q * NT;
                const int i = KC ? e / (TK64 / 2) : 2 * (e % (TS / 2)), k = KC ? 2 * (e % (TK64 / 2)) : e / (TS / 2);
                const bool ok = i < R && k0 + k < K;
                const double* src = KC ? X + (k0 + k) + (long)i * ld : X + i + (long)(k0 + k) * ld;
                cp_async16z(s + (KC ? i * KS64 + k : k * RS + i), ok ? src : X, ok);
            }
        } else {
#pragma unroll
            for (int q = 0; q < TS * TK64 / NT; ++q) {
                const int e = tid + q * NT;
                const int i = KC ? e / TK64 : e % TS, k = KC ? e % TK64 : e / TS;
                const bool ok = i < R && k0 + k < K;
                const double* src = KC ? X + (k0 + k) + (long)i * ld : X + i + (long)(k0 + k) * ld;
                cp_async8(s + (KC ? i * KS64 + k : k * RS + i), ok ? src : X, ok);
            }
        }
    }

    // c += op(A) op(B) over K: op(A) M x K (AK: K-contiguous, A[k + i lda], else
    // A[i + k lda]), op(B) K x N (BK: B[k + j ldb], else B[j + k ldb]).  Starts with
    // the shared memory free and ends with it free for the whole CTA.
    template <bool AK, bool BK>
    static __device__ __forceinline__ void product(Acc& c, Smem& sm, const double* A, long lda, int M, const double* B,
                                                   long ldb, int N, int K, bool va, bool vb) {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        const int g = lane >> 2, t = lane & 3;
        const int wm = (w % WM) * 8 * MI, wn = (w / WM) * 8 * NJ;
        const bool active = wm < M && wn < N;
        const int ns = (K + TK64 - 1) / TK64;
        auto issue = [&](int i, int s) {
            stage<AK>(sm.A[s], A, lda, M, i * TK64, K, va);
            stage<BK>(sm.B[s], B, ldb, N, i * TK64, K, vb);
        };
        if (ns > 0) issue(0, 0);
        cp_async_commit();
        if (ns > 1) issue(1, 1);
        cp_async_commit();
        int s = 0;
        for (int i = 0; i < ns; ++i) {
            cp_async_wait<1>();  // slab i has landed
            __syncthreads();     // for every thread, and all are done with slab i - 1 (stage of slab i + 2)
            const int s2 = s == 0 ? 2 : s - 1;
            if (i + 2 < ns) issue(i + 2, s2);
            cp_async_commit();
            if (active) {
                const double* sA = AK ? sm.A[s] + (wm + g) * KS64 + t : sm.A[s] + t * RS + wm + g;
                const double* sB = BK ? sm.B[s] + (wn + g) * KS64 + t : sm.B[s] + t * RS + wn + g;
#pragma unroll
                for (int k4 = 0; k4 < TK64; k4 += 4) {
                    double a[MI], b[NJ];
#pragma unroll
                    for (int q = 0; q < MI; ++q) a[q] = AK ? sA[8 * q * KS64 + k4] : sA[k4 * RS + 8 * q];
#pragma unroll
                    for (int q = 0; q < NJ; ++q) b[q] = BK ? sB[8 * q * KS64 + k4] : sB[k4 * RS + 8 * q];
#pragma unroll
                    for (int q = 0; q < MI; ++q)
#pragma unroll
                        for (int p = 0; p < NJ; ++p) mma_f64(c.v[q][p], a[q], b[p]);
                }
            }
            s = s == 2 ? 0 : s + 1;
        }
        __syncthreads();
    }
};

// One conditioning step through 64-row tiles (r > 64), one CTA of 256 threads for a
// set of at most 64 columns:
//   V = C - Ua^T Us  (Ua: K x r, ld K; Us: K x N, ld ldu),  U = P V.
// V (ld ldv) is global memory; r even: pair copies.  Ends with a barrier.
__device__ __forceinline__ void cond_tiles(Tile<64>::Smem& sm, int r, const double* Ua, int K, const double* Us, long ldu,
                                           int N, const double* P, const double* C, long ldc, double* V, long ldv,
                                           double* U) {
    using TT = Tile<64>;
    const bool vec = r % 2 == 0;
    if (K > 0 || V != C) {
        for (int r0 = 0; r0 < r; r0 += 64) {
            const int M = min(64, r - r0);
            TT::Acc acc;
            TT::zero(acc);
            TT::add(acc, -1.0, C + r0, ldc, M, N);
            TT::product<true, true>(acc, sm, Ua + (long)r0 * K, K, M, Us, ldu, N, K, vec, vec);
            TT::store(acc, -1.0, V + r0, ldv, M, N);
        }
        __syncthreads();
    }
    for (int r0 = 0; r0 < r; r0 += 64) {
        const int M = min(64, r - r0);
        TT::Acc acc;
        TT::zero(acc);
        // the inverse is lower triangular: rows up to r0 + M - 1
        TT::product<false, true>(acc, sm, P + r0, r, M, V, ldv, N, r0 + M, vec, vec && M % 2 == 0);
        TT::store(acc, 1.0, U + r0, ldu, M, N);
    }
    __syncthreads();
}

}  // namespace mra
