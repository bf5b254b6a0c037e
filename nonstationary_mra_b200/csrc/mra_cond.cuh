// Conditioning steps of the FP64 path (sm_100a): for a set S of at most 64 points
// with a common ancestor a of level j,
//   V = C(Q_a, S) - U_a^T U_{S,0..j-1},   U_{S,j} = L_a^{-1} V,
// the inner loop of the prior levels (S: the knots of sibling regions,
// class_approximation.cpp:84-169) and of the finest level (S: observations,
// ...-loop-regions-at-finest-level-in-prior.cpp:90-200).  One CTA of 4 warps walks
// the chain of ancestors; a step is a stream of 32-deep K slabs (two stages, one
// barrier per slab): the slabs of U_a^T U_S, then L_a^{-1} as one or two more.  V
// stays in shared memory between the two products.
//
// The chain is serial -- barriers, the latency of each step's first slab, the
// Cholesky factorization at its end -- so what keeps the FP64 tensor pipe busy is
// the number of chains per SM, each of which can fill it alone: small CTAs, three
// or four per SM, rather than two large ones (two of 256 threads with three stages:
// prior level of 16,384 regions 12.7 ms, this 10.7).  RC is the tile height (16, 32 or
// 64 >= r): the warps are RC / 16 row groups of 16 rows x column groups that
// share the 64 columns, so that small r multiplies no padding; column fragments
// beyond the set are not computed, and warps stop at the diagonal of triangular
// operands (their row groups rotate with the block index, so that the longest
// does not always fall on the same SM sub-partition).
//
// Operands lie K-contiguous in shared memory, [row][k], 16-byte chunks XORed with
// the row; a lane reads k = 2t and 2t + 1 together (16 bytes) and uses them in two
// consecutive m8n8k4 products, the same permutation of k on both operands.
#pragma once

#include "mra_kernels.cuh"

namespace mra {

constexpr int kCondThreads = 128;

template <int RC>
struct CondSmem {
    static constexpr int CTAS = RC == 64 ? 3 : 4;  // per SM
    static constexpr int PS = RC + 2;              // row stride of a slab [k][row] of L_a^{-1}
    static constexpr int KN = RC < TK64 ? RC : TK64;
    static constexpr int S1 = RC * TK64 > KN * PS ? RC * TK64 : KN * PS;
    static constexpr int AS = 2 * S1 > RC * SLD ? S1 : RC * SLD / 2;
    static constexpr int BS = RC == 64 ? 64 * SLD / 2 : 64 * TK64;
    double A[2][AS];  // two stages; also the matrix of the Cholesky factorization (RC x SLD)
    double B[2][BS];  // two stages; also V [column][row] and the inverse of the factor
    double red[kCondThreads / 32];
    int flag;
};

// One step's operands.  EVEN kernels need r even (then every operand row is
// 16-byte aligned and is copied in pairs).
struct CondOp {
    const double* Ua;  // K x r, ld K
    int K;
    const double* Us;  // rows 0..K-1 of the set's U, ld ldu
    long ldu;
    int N;
};

__device__ __forceinline__ int cond_swz(int row) { return ((row & 1) << 2) | ((row >> 1) & 3); }
// sign flips on the integer pipe
__device__ __forceinline__ double2 neg2(double2 v) {
    return make_double2(__hiloint2double(__double2hiint(v.x) ^ (int)0x80000000, __double2loint(v.x)),
                        __hiloint2double(__double2hiint(v.y) ^ (int)0x80000000, __double2loint(v.y)));
}
__device__ __forceinline__ double2 lds2(const double* p) { return *reinterpret_cast<const double2*>(p); }

template <int RC, bool EVEN>
struct Cond {
    static constexpr int RW = RC / 16, CW = 4 / RW, NF = 8 / CW;  // row groups, column groups, fragments per warp
    static constexpr int NP = RC > TK64 ? 2 : 1;                  // slabs of L_a^{-1}
    static constexpr int KN = RC < TK64 ? RC : TK64;              // their depth
    static constexpr int PS = CondSmem<RC>::PS;
    static constexpr int VC = RC > TK64 ? 32 : 64;                // columns of V per stage
    using Smem = CondSmem<RC>;

    Smem& sm;
    int r;
    int wr, wc;  // this warp's row group and column group
    int g, t;

    __device__ __forceinline__ Cond(Smem& s, int r_) : sm(s), r(r_) {
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
        wr = (w + blockIdx.x) % RW;
        wc = w / RW;
        g = lane >> 2;
        t = lane & 3;
    }

    // rows x 32 elements of K-contiguous rows (row i at X + i ld) from k0, into [row][k]
    __device__ __forceinline__ void load_rows(double* s, const double* X, long ld, int rows, int pad, int k0, long K) {
        const int tid = threadIdx.x;
        constexpr int PK = EVEN ? 16 : 32, NR = kCondThreads / PK;  // copies per row, rows at once
        const int c = tid % PK;
        const long k = k0 + (EVEN ? 2 * c : c);
        const double* src = X + k + (long)(tid / PK) * ld;
        for (int i = tid / PK; i < pad; i += NR, src += NR * ld) {
            const bool ok = i < rows && k < K;
            double* dst = s + i * TK64 + (EVEN ? (c ^ cond_swz(i)) * 2 : ((c >> 1) ^ cond_swz(i)) * 2 + (c & 1));
            if (EVEN) cp_async16z(dst, ok ? src : X, ok);
            else cp_async8(dst, ok ? src : X, ok);
        }
    }
    // slab q of L_a^{-1}: [k][row]
    __device__ __forceinline__ void load_inv(const double* P, int q, double* s) {
        constexpr int PR = EVEN ? RC / 2 : RC;
        for (int e = threadIdx.x; e < PR * KN; e += kCondThreads) {
            const int i = (EVEN ? 2 : 1) * (e % PR), kk = e / PR, k = q * TK64 + kk;
            const bool ok = i < r && k < r;
            const double* src = ok ? P + i + (long)k * r : P;
            if (EVEN) cp_async16z(s + kk * PS + i, src, ok);
            else cp_async8(s + kk * PS + i, src, ok);
        }
    }

    // acc -= A B over one slab, F column fragments; A: this warp's 16 rows
    template <int F>
    __device__ __forceinline__ void mma_slab(double (&acc)[2][NF][2], const double* sA, const double* sB) const {
        const int off0 = ((cond_swz(g) & 4) | (t ^ (cond_swz(g) & 3))) * 2;
        const double* a0 = sA + (16 * wr + g) * TK64;
        const double* b0 = sB + (8 * wc + g) * TK64;
#pragma unroll 2
        for (int s = 0; s < 4; ++s) {
            const int off = off0 ^ (8 * s);
            const double2 x0 = neg2(lds2(a0 + off)), x1 = neg2(lds2(a0 + 8 * TK64 + off));
            double2 y[F];
#pragma unroll
            for (int f = 0; f < F; ++f) y[f] = lds2(b0 + f * CW * 8 * TK64 + off);
#pragma unroll
            for (int f = 0; f < F; ++f) {
                mma_f64(acc[0][f], x0.x, y[f].x);
                mma_f64(acc[1][f], x1.x, y[f].x);
            }
#pragma unroll
            for (int f = 0; f < F; ++f) {
                mma_f64(acc[0][f], x0.y, y[f].y);
                mma_f64(acc[1][f], x1.y, y[f].y);
            }
        }
    }
    __device__ __forceinline__ void mma_slab_n(int nf, double (&acc)[2][NF][2], const double* sA, const double* sB) const {
        // widths 1, 2, 4, 6, 8 only (uniform in the warp): the code of all eight did not stay in the instruction
        // cache; the extra fragment's columns are never stored
        if (nf == 1) mma_slab<1>(acc, sA, sB);
        else if (nf == 2) mma_slab<2>(acc, sA, sB);
        else if constexpr (NF > 2) {
            if (nf > 6) { if constexpr (NF >= 8) mma_slab<8>(acc, sA, sB); }
            else if (nf > 4) { if constexpr (NF >= 6) mma_slab<6>(acc, sA, sB); }
            else if (nf > 2) mma_slab<4>(acc, sA, sB);
        }
    }
    // acc += P V over slab q of L_a^{-1} (rows in pairs: fragment i holds rows 16 wr + 2 g + i), F column fragments
    template <int F>
    __device__ __forceinline__ void mma_inv(double (&acc)[2][NF][2], const double* sP, int q, int steps) const {
        const int sw = cond_swz(g);
        const double* a0 = sP + 2 * t * PS + 16 * wr + 2 * g;
#pragma unroll 1
        for (int s = 0; s < steps; ++s) {
            const double2 x0 = lds2(a0 + 8 * s * PS), x1 = lds2(a0 + (8 * s + 1) * PS);
            const int off = ((q * (TK64 / 2) + 4 * s + t) ^ sw) * 2;
            double2 y[F];
#pragma unroll
            for (int f = 0; f < F; ++f) {
                const int c = (f * CW + wc) * 8;
                y[f] = lds2(sm.B[c / VC] + (c % VC + g) * RC + off);
            }
#pragma unroll
            for (int f = 0; f < F; ++f) {
                mma_f64(acc[0][f], x0.x, y[f].x);
                mma_f64(acc[1][f], x0.y, y[f].x);
            }
#pragma unroll
            for (int f = 0; f < F; ++f) {
                mma_f64(acc[0][f], x1.x, y[f].y);
                mma_f64(acc[1][f], x1.y, y[f].y);
            }
        }
    }
    __device__ __forceinline__ void mma_inv_n(int nf, double (&acc)[2][NF][2], const double* sP, int q, int steps) const {
        if (nf == 1) mma_inv<1>(acc, sP, q, steps);
        else if (nf == 2) mma_inv<2>(acc, sP, q, steps);
        else if constexpr (NF > 2) {
            if (nf > 6) { if constexpr (NF >= 8) mma_inv<8>(acc, sP, q, steps); }
            else if (nf > 4) { if constexpr (NF >= 6) mma_inv<6>(acc, sP, q, steps); }
            else if (nf > 2) mma_inv<4>(acc, sP, q, steps);
        }
    }
    // column fragments (f CW + wc) 8 < N of this warp
    __device__ __forceinline__ int frags(int N) const { return ((N + 7) / 8 - wc + CW - 1) / CW; }

    // acc = C (r x N, ld ldc)
    __device__ __forceinline__ void init(double (&acc)[2][NF][2], const double* C, long ldc, int N) const {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int row = 16 * wr + 8 * i + g;
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const int c = (f * CW + wc) * 8 + 2 * t;
#pragma unroll
                for (int h = 0; h < 2; ++h) acc[i][f][h] = (row < r && c + h < N) ? C[row + (long)(c + h) * ldc] : 0.0;
            }
        }
    }

    // U = P (C - Ua^T Us); C: r x N, ld ldc; V (may be null): r x N, ld ldu; U: ld ldu.
    // Starts with the shared memory free, ends with a barrier.
    __device__ __forceinline__ void step(const CondOp& o, const double* P, const double* C, long ldc, double* V, double* U) {
        const int N = o.N, N8 = (N + 7) & ~7;
        const bool act = 16 * wr < r;
        const int nf = act ? frags(N) : 0;
        const int ns = (o.K + TK64 - 1) / TK64;
        double acc[2][NF][2];
        auto issue = [&](int v) {  // slab v of the operands; after the last, slab 0 of L_a^{-1}
            if (v < ns) {
                load_rows(sm.A[v & 1], o.Ua, o.K, r, RC, v * TK64, o.K);
                load_rows(sm.B[v & 1], o.Us, o.ldu, N, N8, v * TK64, o.K);
            } else {
                load_inv(P, 0, sm.A[v & 1]);
            }
            cp_async_commit();
        };
        issue(0);
        init(acc, C, ldc, N);
        for (int i = 0; i < ns; ++i) {
            cp_async_wait<0>();  // slab i has landed
            __syncthreads();     // for every thread, and all are done with slab i - 1 (the other stage)
            issue(i + 1);
            mma_slab_n(nf, acc, sm.A[i & 1], sm.B[i & 1]);
        }
        __syncthreads();
        if (NP > 1) load_inv(P, 1, sm.A[(ns + 1) & 1]);
        cp_async_commit();
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const int c = (f * CW + wc) * 8 + 2 * t;
            if (f >= nf) continue;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int row = 16 * wr + 8 * i + g;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double v = acc[i][f][h];
                    sm.B[c / VC][(c % VC + h) * RC + (((row >> 1) ^ cond_swz(2 * t + h)) << 1) + (row & 1)] = v;
                    if (V && row < r && c + h < N) V[row + (long)(c + h) * o.ldu] = v;
                    acc[i][f][h] = 0.0;
                }
            }
        }
        // rows 16 wr .. 16 wr + 15 of a lower-triangular factor end at column 16 wr + 15
        const int end = (16 * (wr + 1) < r ? 16 * (wr + 1) : r + 7) / 8;
        cp_async_wait<1>();
        __syncthreads();
        mma_inv_n(nf, acc, sm.A[ns & 1], 0, end < KN / 8 ? end : KN / 8);
        if (NP > 1) {
            cp_async_wait<0>();
            __syncthreads();
            if (end > TK64 / 8) mma_inv_n(nf, acc, sm.A[(ns + 1) & 1], 1, end - TK64 / 8);
        }
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const int c = (f * CW + wc) * 8 + 2 * t, row = 16 * wr + 2 * g;
            if (f >= nf) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (c + h >= N) continue;
                double* u = U + row + (long)(c + h) * o.ldu;
                if (EVEN) {
                    if (row < r) *reinterpret_cast<double2*>(u) = make_double2(acc[0][f][h], acc[1][f][h]);
                } else {
                    if (row < r) u[0] = acc[0][f][h];
                    if (row + 1 < r) u[1] = acc[1][f][h];
                }
            }
        }
        __syncthreads();
    }
};

}  // namespace mra
