// Finest level of the MRA hot path (...-loop-regions-at-finest-level-in-prior.cpp:
// 90-269, class_approximation.cpp:52-82): conditioning of the observations on
// their ancestors, the finest regions' conditional covariances with their
// Cholesky factors, and the log-likelihood terms.
//
// The level runs as separate launches, each split by what is independent in it,
// so that neither a few heavily clustered regions nor a tree with few regions
// leaves the chip to a handful of CTAs (one CTA per level M-3 region with all of
// these steps inside took 2.43 of the 2.61 ms of an 8,192-point evaluation,
// 16 CTAs in flight, and 79 of 93 ms of a 262,144-point clustered prediction,
// one CTA finishing the largest regions):
//   k_cov_set               C(Q_{a_j}, S) of every ancestor level, into B^
//   k_condition_set         V_j and U_j of a chunk of at most 64 observations:
//                           every observation conditions on its own, so the
//                           chunks are as many as the chip needs
//                           (k_finest_condition_any: r > 64 and FP32 storage)
//   (mra_small.cu)          Sigma, L_Sigma, y~, B^ of finest regions of at most 64
//                           observations, sibling groups of small ones together
//                           with their parent's posterior
//   k_heavy_*               the same of larger finest regions in 64 x 64 tiles,
//                           one CTA per tile, the block columns in turn
//   k_finest_terms          log-lik terms summed per sibling group
#include "mra_cond.cuh"
#include "mra_tile.cuh"

namespace mra {

// ---------------------------------------------------------------------------
// covariance of the observations with their ancestors' knots
// ---------------------------------------------------------------------------
// (CondSet: the observations, or the prediction points, of every sub-tree in chunks.)
// Task (chunk, j): block C(Q_{a_j}, S_chunk), r x n, into row block j of B^.  The
// deepest ancestor (level M-2) differs between the sibling groups of a chunk.
// Issue-bound like k_cov_level: its own launch keeps 4 CTAs per SM busy.
template <typename T, int KIND>
__global__ void __launch_bounds__(kCovThreads, 4) k_cov_set(Geom g, DevTree<T> t, CondSetT<T> set) {
    constexpr int CH = sizeof(T) == 8 ? kCovChunk : 96;  // FP32: the chunk of fill_cov, and so its compiled code
    __shared__ __align__(16) double stage[7 * CH];
    const int r = t.r, L = t.L, m = t.M - 2;
    const long Lr = (long)L * r;
    const long ntask = set.n * L;
    for (long b = blockIdx.x; b < ntask; b += gridDim.x) {
        const long q = (unsigned)b / (unsigned)L;  // at most 2^31 tasks
        const int j = (int)(b - q * L);
        const FinChunk ch = set.chunks[q];
        const long unit = ch.unit;  // local index at level M-3 (0 when M == 2)
        if (skipped(t, chunk_region(t, unit))) continue;
        if (j < m) {
            const long a = ancestor(t, m - 1, unit, j);
            cov_block<T, KIND, CH>(g, t.pts, a * r, r, set.pt0 + ch.lo, ch.n, false, set.V + ch.lo * Lr + (long)j * r, Lr,
                               stage);
        } else {
            const long g0 = m > 0 ? unit * t.J : 0, g1 = m > 0 ? g0 + t.J : 1;
            const long s2 = t.lstart[m];
            for (long gl = g0; gl < g1; ++gl) {
                const long glo = set.glo[gl], ghi = set.ghi[gl];
                const long lo = glo > ch.lo ? glo : ch.lo, hi = ghi < ch.lo + ch.n ? ghi : ch.lo + ch.n;
                if (lo >= hi) continue;
                cov_block<T, KIND, CH>(g, t.pts, (s2 + gl) * r, r, set.pt0 + lo, (int)(hi - lo), false,
                                   set.V + lo * Lr + (long)m * r, Lr, stage);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// conditioning: V_j = C_j - U_{a_j}^T U_{S,0..j-1},  U_{S,j} = L_{a_j}^{-1} V_j
// ---------------------------------------------------------------------------
// FP64, r <= RC <= 64 (mra_cond.cuh): one CTA per chunk.
template <int RC, bool EVEN>
__global__ void __launch_bounds__(kCondThreads, CondSmem<RC>::CTAS) k_condition_set(DevTree<double> t, CondSet set) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    const int r = t.r, L = t.L, m = t.M - 2;
    const long rr = (long)r * r, Lr = (long)L * r;
    const FinChunk ch = set.chunks[blockIdx.x];
    const long unit = ch.unit;
    if (skipped(t, chunk_region(t, unit))) return;
    Cond<RC, EVEN> cond(*reinterpret_cast<CondSmem<RC>*>(la_dyn_smem), r);
    double* V = set.V + ch.lo * Lr;
    double* U = set.U + ch.lo * Lr;
    // levels 0..M-3, then level M-2 per sibling group of the chunk; one call of
    // step, whose code then stays in the instruction cache
    const int ng = m > 0 ? t.J : 1;
    const long g0 = m > 0 ? unit * t.J : 0, s2 = t.lstart[m];
    for (int s = 0; s < m + ng; ++s) {
        long a, lo = ch.lo, hi = ch.lo + ch.n;
        const int j = s < m ? s : m;
        if (s < m) {
            a = ancestor(t, m - 1, unit, j);
        } else {
            a = s2 + g0 + (s - m);
            if (set.glo[a - s2] > lo) lo = set.glo[a - s2];
            if (set.ghi[a - s2] < hi) hi = set.ghi[a - s2];
            if (lo >= hi) continue;
        }
        const long d = (lo - ch.lo) * Lr;
        const CondOp o{t.U + t.u_off[j] + (a - t.lstart[j]) * (long)j * rr, j * r, U + d, Lr, (int)(hi - lo)};
        double* Vj = V + d + (long)j * r;
        cond.step(o, t.Pinv + a * rr, Vj, Lr, Vj, U + d + (long)j * r);
    }
}

// The same through 64-row tiles (FP64, r > 64) or the general products (FP32 storage).
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_finest_condition_any(DevTree<T> t) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    const int r = t.r, L = t.L, m = t.M - 2;
    const long rr = (long)r * r, Lr = (long)L * r;
    const FinChunk ch = t.chunks[blockIdx.x];
    const long unit = ch.unit;
    if (skipped(t, chunk_region(t, unit))) return;
    auto step = [&](long a, int j, const T* Ua, long d, int n) {
        T* V = t.Bhat + (ch.lo + d) * Lr + (long)j * r;
        T* U = t.Ufin + (ch.lo + d) * Lr;
        if constexpr (sizeof(T) == 8) {
            cond_tiles(*reinterpret_cast<Tile<64>::Smem*>(la_dyn_smem), r, Ua, j * r, U, Lr, n, t.Pinv + a * rr, V, Lr, V, Lr,
                       U + (long)j * r);
        } else {
            LaSmem<T>& sm = la_smem<T>();
            if (j > 0) gemm<T, true, false>(r, n, j * r, (T)-1, Ua, (long)j * r, U, Lr, (T)1, V, Lr, sm);
            gemm<T, false, false>(r, n, r, (T)1, t.Pinv + a * rr, r, V, Lr, (T)0, U + (long)j * r, Lr, sm);
        }
    };
    const long g0 = m > 0 ? unit * t.J : 0, g1 = m > 0 ? g0 + t.J : 1;
    const long s2 = t.lstart[m];
    long gl = g0 - 1;
    for (int j = 0; j < m || gl + 1 < g1;) {
        long a, lo = ch.lo, hi = ch.lo + ch.n;
        const T* Ua;
        int jj;
        if (j < m) {
            jj = j++;
            a = ancestor(t, m - 1, unit, jj);
            Ua = t.U + t.u_off[jj] + (a - t.lstart[jj]) * (long)jj * rr;
        } else {
            ++gl;
            jj = m;
            a = s2 + gl;
            if (t.sub_lo[a] > lo) lo = t.sub_lo[a];
            if (t.sub_hi[a] < hi) hi = t.sub_hi[a];
            if (lo >= hi) continue;
            Ua = t.U + t.u_off[m] + gl * (long)m * rr;
        }
        step(a, jj, Ua, lo - ch.lo, (int)(hi - lo));
    }
}

// ---------------------------------------------------------------------------
// finest regions in FP32 storage (mixed path): one CTA per region, from a queue,
// most expensive first
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads, 2) k_finest_regions_f32(Geom g, DevTree<float> t) {
    LaSmem<float>& sm = la_smem<float>();
    __shared__ long s_u;
    const int L = t.L;
    const long Lr = (long)L * t.r;
    const long cnt2 = level_count(t.J, t.M - 2);
    for (;;) {
        if (threadIdx.x == 0) {
            int q = atomicAdd(&t.queue[0], 1);
            s_u = q < t.n_fin_items ? t.fin_items[q] : -1;
        }
        __syncthreads();
        const long item = s_u;
        __syncthreads();
        if (item < 0) break;
        const long c = item - cnt2;
        if (skipped(t, (long)t.fin_anc[c * L + L - 1])) continue;
        const long o0 = t.obs_off[c];
        const int n = (int)(t.obs_off[c + 1] - o0);
        float* S = t.Lsig + t.lsig_off[c];
        fill_cov<float>(g, t.pts, t.obs0 + o0, n, t.obs0 + o0, n, true, S, n, sm);
        __syncthreads();
        gemm<float, true, false>(n, n, (int)Lr, -1.f, t.Ufin + o0 * Lr, Lr, t.Ufin + o0 * Lr, Lr, 1.f, S, n, sm);
        double ld = 0.0;
        int info = potrf_lower<float>(n, S, n, sm, &ld);
        double* ytc = t.yt + o0;
        for (int e = threadIdx.x; e < n; e += kThreads) ytc[e] = t.y[o0 + e];
        __syncthreads();
        trsv_lower_f64<float>(n, S, n, ytc);
        trsm_right_lower_trans<float>((int)Lr, n, S, n, t.Bhat + o0 * Lr, Lr, sm);
        double part = 0.0;
        for (int e = threadIdx.x; e < n; e += kThreads) part += ytc[e] * ytc[e];
        double yy = cta_sum(part, sm);
        if (threadIdx.x == 0) {
            t.dchild[c] = yy + ld;
            if (info) report_error(t.err, t.n_int + c);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// finest regions of more than 64 observations (FP64), in 64 x 64 tiles
// ---------------------------------------------------------------------------
// One CTA per tile throughout, on the tile products of mra_tile.cuh (8-byte copies
// where a region's odd size leaves its columns unaligned).
__device__ __forceinline__ bool aligned16(const double* p, long ld) {
    return ((unsigned long)p & 15ul) == 0 && ld % 2 == 0;
}

// C(S, S) into Sigma's lower tiles.
template <int KIND>
__global__ void __launch_bounds__(kCovThreads, 4) k_cov_heavy(Geom g, DevTree<double> t) {
    __shared__ __align__(16) double stage[7 * kCovChunk];
    const HeavyTile ht = t.heavy_tiles[blockIdx.x];
    const long c = t.heavy[ht.h];
    if (skipped(t, (long)t.fin_anc[c * t.L + t.L - 1])) return;
    const long o0 = t.obs_off[c];
    const int n = (int)(t.obs_off[c + 1] - o0);
    const int i0 = 64 * ht.bi, j0 = 64 * ht.bj;
    cov_block<double, KIND>(g, t.pts, t.obs0 + o0 + i0, min(64, n - i0), t.obs0 + o0 + j0, min(64, n - j0),
                            ht.bi == ht.bj, t.Lsig + t.lsig_off[c] + i0 + (long)j0 * n, n, stage);
}

// Sigma = C - U_S^T U_S, lower tiles.
__global__ void __launch_bounds__(kThreads, 2) k_heavy_sigma(DevTree<double> t) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using TT = Tile<64>;
    TT::Smem& sm = *reinterpret_cast<TT::Smem*>(la_dyn_smem);
    const long Lr = (long)t.L * t.r;
    const HeavyTile ht = t.heavy_tiles[blockIdx.x];
    const long c = t.heavy[ht.h];
    if (skipped(t, (long)t.fin_anc[c * t.L + t.L - 1])) return;
    const long o0 = t.obs_off[c];
    const int n = (int)(t.obs_off[c + 1] - o0);
    const int i0 = 64 * ht.bi, j0 = 64 * ht.bj;
    const int ni = min(64, n - i0), nj = min(64, n - j0);
    double* S = t.Lsig + t.lsig_off[c] + i0 + (long)j0 * n;
    const bool vec = Lr % 2 == 0;
    TT::Acc acc;
    TT::zero(acc);
    TT::add(acc, -1.0, S, n, ni, nj);
    TT::product<true, true>(acc, sm, t.Ufin + (o0 + i0) * Lr, Lr, ni, t.Ufin + (o0 + j0) * Lr, Lr, nj, (int)Lr, vec, vec);
    TT::store(acc, -1.0, S, n, ni, nj);
}

// Left-looking block column k of the factorization of [Sigma; V]: the tiles of
// the block column (rows k.. of Sigma, then the row tiles of V) subtract the
// product of what is already factored; the diagonal tile is then factored and
// inverted, and y~_k solved.  blockIdx.x = region * tiles + tile.
__global__ void __launch_bounds__(kThreads, 2) k_heavy_column(DevTree<double> t, int k, int tiles) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using TT = Tile<64>;
    TT::Smem& tm = *reinterpret_cast<TT::Smem*>(la_dyn_smem);
    const long Lr = (long)t.L * t.r;
    const int h = blockIdx.x / tiles, tile = blockIdx.x % tiles;
    const long c = t.heavy[h];
    if (skipped(t, (long)t.fin_anc[c * t.L + t.L - 1])) return;
    const long o0 = t.obs_off[c];
    const int n = (int)(t.obs_off[c + 1] - o0);
    const int rows = (n + 63) / 64 - k;  // row tiles of Sigma in this block column
    const int j0 = 64 * k, nj = min(64, n - j0);
    double* S = t.Lsig + t.lsig_off[c];
    const bool vs = aligned16(S, n);
    const bool inV = tile >= rows;
    const long x0 = 64L * (tile - rows);
    if (inV && x0 >= Lr) return;
    const int i0 = j0 + 64 * tile;
    double* A = inV ? t.Bhat + o0 * Lr + x0 : S + i0;  // factored columns 0..j0-1 of the row tile
    const long lda = inV ? Lr : n;
    const int ni = inV ? (int)min(64L, Lr - x0) : min(64, n - i0);
    double* W = A + (long)j0 * lda;
    if (k > 0) {
        TT::Acc acc;
        TT::zero(acc);
        TT::add(acc, -1.0, W, lda, ni, nj);
        // a pair copy starts at an even row: the valid rows must be even, or rows beyond the tile be readable
        TT::product<false, false>(acc, tm, A, lda, ni, S + j0, n, nj, j0, (inV ? Lr % 2 == 0 : vs) && ni % 2 == 0,
                                  vs && nj % 2 == 0);
        TT::store(acc, -1.0, W, lda, ni, nj);
        __syncthreads();
    }
    if (inV || tile > 0) return;
    LaSmem<double>& sm = la_smem<double>();
    double* X = t.heavy_inv + (long)h * 64 * 64;
    double ld = 0.0;
    const int info = potrf_small(nj, W, n, sm, &ld, X, 64);
    // y~_k = X (y_k - L_(k,0..k-1) y~_(0..k-1)): 4 threads per row over the columns, 16 loads
    // in flight (4: a late block column of a region of 450 takes 66 us instead of 41; an
    // evaluation whose largest region holds 522 observations 3.58 ms instead of 3.53)
    double* yt = t.yt + o0;
    double* part = &sm.A[0][0];
    {
        const int q = threadIdx.x & 63, cg = threadIdx.x >> 6;
        double s = 0.0;
        if (q < nj) {
#pragma unroll 16
            for (int x = cg; x < j0; x += 4) s += S[j0 + q + (long)x * n] * yt[x];
        }
        part[threadIdx.x] = s;
        __syncthreads();
        if (threadIdx.x < nj) {
            const int e = threadIdx.x;
            yt[j0 + e] = t.y[o0 + j0 + e] - ((part[e] + part[64 + e]) + (part[128 + e] + part[192 + e]));
        }
        __syncthreads();
    }
    trmv_lower_inv<double>(nj, X, 64, yt + j0, yt + j0);
    double p2 = 0.0;
    for (int e = threadIdx.x; e < nj; e += kThreads) p2 += yt[j0 + e] * yt[j0 + e];
    const double yy = cta_sum(p2, sm);
    if (threadIdx.x == 0) {
        t.dchild[c] = (k == 0 ? 0.0 : t.dchild[c]) + yy + ld;
        if (info) report_error(t.err, t.n_int + c);
    }
}

// The tiles below the diagonal of block column k (and V's) times L_kk^{-T}, in place.
__global__ void __launch_bounds__(kThreads, 2) k_heavy_panel(DevTree<double> t, int k, int tiles) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using TT = Tile<64>;
    TT::Smem& sm = *reinterpret_cast<TT::Smem*>(la_dyn_smem);
    const long Lr = (long)t.L * t.r;
    const int h = blockIdx.x / tiles, tile = blockIdx.x % tiles;
    const long c = t.heavy[h];
    if (skipped(t, (long)t.fin_anc[c * t.L + t.L - 1])) return;
    const long o0 = t.obs_off[c];
    const int n = (int)(t.obs_off[c + 1] - o0);
    const int rows = (n + 63) / 64 - k - 1;  // row tiles of Sigma below the diagonal
    const int j0 = 64 * k, nj = min(64, n - j0);
    const double* X = t.heavy_inv + (long)h * 64 * 64;
    double* W;
    long ldw;
    int ni;
    if (tile < rows) {
        const int i0 = j0 + 64 * (tile + 1);
        W = t.Lsig + t.lsig_off[c] + i0 + (long)j0 * n;
        ldw = n;
        ni = min(64, n - i0);
    } else {
        const long x0 = 64L * (tile - rows);
        if (x0 >= Lr) return;
        W = t.Bhat + (o0 + j0) * Lr + x0;
        ldw = Lr;
        ni = (int)min(64L, Lr - x0);
    }
    TT::Acc acc;
    TT::zero(acc);
    TT::product<false, false>(acc, sm, W, ldw, ni, X, 64, nj, nj, aligned16(W, ldw) && ni % 2 == 0, nj % 2 == 0);
    TT::store(acc, 1.0, W, ldw, ni, nj);
}

// ---------------------------------------------------------------------------
// finest regions of more than 64 observations, FP32 storage
// ---------------------------------------------------------------------------
// potrf_blocked<float> and trsm_right_lower_trans<float> of a region spread over
// the chip: per 16-wide panel, every element goes through the same operations in
// the same order as in one CTA (FP64 diagonal block and panel solves, one rounded
// FP32 update per panel), so the results are bitwise the same.  Two launches per
// panel b:
//   k_heavy32_panel   L's diagonal block b and the rows below it (each CTA factors
//                     the 16 x 16 block for itself); V's update by panel b - 1
//   k_heavy32_update  Sigma's lower tiles minus panel b's products; V's columns of
//                     panel b; the factored diagonal block into place
// A clustered 65,536-point evaluation spent 6.3 of 11 ms in one CTA's largest
// region (394 observations); it takes 6.9 ms now.
struct Heavy32 {
    float* S;    // Sigma, n x n
    float* V;    // B^ rows: Lr x n, ld Lr
    float* D;    // 16 x 16 diagonal block of the current panel, factored (column-major)
    double* ld;  // running log-determinant
    long c;
    int n;
};
__device__ __forceinline__ Heavy32 heavy32(const DevTree<float>& t, int h) {
    Heavy32 r;
    r.c = t.heavy[h];
    const long o0 = t.obs_off[r.c];
    r.n = (int)(t.obs_off[r.c + 1] - o0);
    r.S = t.Lsig + t.lsig_off[r.c];
    r.V = t.Bhat + o0 * (long)t.L * t.r;
    r.D = reinterpret_cast<float*>(t.heavy_inv + (long)h * 64 * 64);
    r.ld = t.heavy_inv + (long)h * 64 * 64 + 128;
    return r;
}

__global__ void __launch_bounds__(kThreads, 2) k_heavy32_sigma(Geom g, DevTree<float> t) {
    LaSmem<float>& sm = la_smem<float>();
    const long Lr = (long)t.L * t.r;
    const HeavyTile ht = t.heavy_tiles[blockIdx.x];
    const Heavy32 r = heavy32(t, ht.h);
    const long o0 = t.obs_off[r.c];
    const int i0 = 64 * ht.bi, j0 = 64 * ht.bj;
    const int ni = min(64, r.n - i0), nj = min(64, r.n - j0);
    float* S = r.S + i0 + (long)j0 * r.n;
    fill_cov<float>(g, t.pts, t.obs0 + o0 + i0, ni, t.obs0 + o0 + j0, nj, ht.bi == ht.bj, S, r.n, sm);
    __syncthreads();
    gemm<float, true, false>(ni, nj, (int)Lr, -1.f, t.Ufin + (o0 + i0) * Lr, Lr, t.Ufin + (o0 + j0) * Lr, Lr, 1.f, S, r.n,
                             sm);
}

// tasks per region: cs row chunks of 256, then xt x ct tiles of V
__global__ void __launch_bounds__(kThreads, 2) k_heavy32_panel(DevTree<float> t, int b, int cs, int ct, int tasks) {
    LaSmem<float>& sm = la_smem<float>();
    const int tid = threadIdx.x;
    const Heavy32 r = heavy32(t, blockIdx.x / tasks);
    int task = blockIdx.x % tasks;
    const int n = r.n, b0 = 16 * b, nb = min(NB, n - b0), rest = n - b0 - nb;
    const long lda = n;
    if (task >= cs) {  // V(:, b0..) -= V(:, panel b - 1) L(b0.., panel b - 1)^T
        task -= cs;
        const long Lr = (long)t.L * t.r, x0 = 64L * (task / ct);
        const int c0 = b0 + 64 * (task % ct), p0 = b0 - NB;
        if (c0 >= n) return;
        gemm<float, false, true>((int)min(64L, Lr - x0), min(64, n - c0), NB, -1.f, r.V + x0 + p0 * Lr, Lr,
                                 r.S + c0 + p0 * lda, lda, 1.f, r.V + x0 + c0 * Lr, Lr, sm);
        return;
    }
    if (task > 0 && 256 * task >= rest) return;
    for (int e = tid; e < nb * nb; e += kThreads) {
        int i = e % nb, j = e / nb;
        sm.D[i][j] = (double)r.S[(b0 + i) + (long)(b0 + j) * lda];
    }
    if (tid == 0) sm.flag = 0;
    __syncthreads();
    if (tid < 32) {
        const int lane = tid;
        for (int k = 0; k < nb; ++k) {
            if (lane == 0) {
                double d = sm.D[k][k];
                if (!(d > 0.0) && sm.flag == 0) sm.flag = b0 + k + 1;
                double sq = sqrt(d);
                sm.D[k][k] = sq;
                sm.inv[k] = 1.0 / sq;
            }
            __syncwarp();
            if (lane > k && lane < nb) sm.D[lane][k] *= sm.inv[k];
            __syncwarp();
            if (lane > k && lane < nb) {
                const double lik = sm.D[lane][k];
                for (int j = k + 1; j <= lane; ++j) sm.D[lane][j] -= lik * sm.D[j][k];
            }
            __syncwarp();
        }
    }
    __syncthreads();
    if (task == 0) {
        for (int e = tid; e < nb * nb; e += kThreads) {
            int i = e % nb, j = e / nb;
            r.D[e] = j <= i ? (float)sm.D[i][j] : 0.f;
        }
        if (tid == 0) {
            double ld = b == 0 ? 0.0 : *r.ld;
            for (int k = 0; k < nb; ++k) ld += 2.0 * log(sm.D[k][k]);
            *r.ld = ld;
            if (sm.flag) report_error(t.err, t.n_int + r.c);
        }
    }
    for (int row = 256 * task + tid; row < min(rest, 256 * (task + 1)); row += kThreads) {
        double x[NB];
        float* p = r.S + (b0 + nb + row) + (long)b0 * lda;
#pragma unroll
        for (int i = 0; i < NB; ++i) x[i] = i < nb ? (double)p[(long)i * lda] : 0.0;
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            if (i < nb) {
                double s = x[i];
#pragma unroll
                for (int k = 0; k < i; ++k) s -= sm.D[i][k] * x[k];
                x[i] = s * sm.inv[i];
            }
        }
#pragma unroll
        for (int i = 0; i < NB; ++i)
            if (i < nb) p[(long)i * lda] = (float)x[i];
    }
}

// tasks per region: cv row chunks of V, then the lower tiles of the trailing matrix
__global__ void __launch_bounds__(kThreads, 2) k_heavy32_update(DevTree<float> t, int b, int cv, int tasks) {
    LaSmem<float>& sm = la_smem<float>();
    const int tid = threadIdx.x;
    const Heavy32 r = heavy32(t, blockIdx.x / tasks);
    int task = blockIdx.x % tasks;
    const int n = r.n, b0 = 16 * b, nb = min(NB, n - b0), rest = n - b0 - nb;
    const long lda = n;
    if (task >= cv) {
        task -= cv;
        int ti = 0;
        while ((ti + 1) * (ti + 2) / 2 <= task) ++ti;
        const int tj = task - ti * (ti + 1) / 2;
        if (64 * ti >= rest) return;
        const float* P = r.S + (b0 + nb) + (long)b0 * lda;
        gemm<float, false, true>(min(64, rest - 64 * ti), min(64, rest - 64 * tj), nb, -1.f, P + 64 * ti, lda, P + 64 * tj,
                                 lda, 1.f, r.S + (b0 + nb + 64 * ti) + (long)(b0 + nb + 64 * tj) * lda, lda, sm);
        return;
    }
    if (task == 0)
        for (int e = tid; e < nb * nb; e += kThreads) r.S[(b0 + e % nb) + (long)(b0 + e / nb) * lda] = r.D[e];
    for (int e = tid; e < nb * nb; e += kThreads) sm.D[e % nb][e / nb] = (double)r.D[e];
    __syncthreads();
    if (tid < nb) sm.inv[tid] = 1.0 / sm.D[tid][tid];
    __syncthreads();
    const long Lr = (long)t.L * t.r;
    for (long row = 256L * task + tid; row < min(Lr, 256L * (task + 1)); row += kThreads) {
        double x[NB];
        float* p = r.V + row + (long)b0 * Lr;
#pragma unroll
        for (int i = 0; i < NB; ++i) x[i] = i < nb ? (double)p[(long)i * Lr] : 0.0;
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            if (i < nb) {
                double s = x[i];
#pragma unroll
                for (int k = 0; k < i; ++k) s -= sm.D[i][k] * x[k];
                x[i] = s * sm.inv[i];
            }
        }
#pragma unroll
        for (int i = 0; i < NB; ++i)
            if (i < nb) p[(long)i * Lr] = (float)x[i];
    }
}

__global__ void __launch_bounds__(kThreads, 2) k_heavy32_terms(DevTree<float> t) {
    LaSmem<float>& sm = la_smem<float>();
    const Heavy32 r = heavy32(t, blockIdx.x);
    const long o0 = t.obs_off[r.c];
    double* ytc = t.yt + o0;
    for (int e = threadIdx.x; e < r.n; e += kThreads) ytc[e] = t.y[o0 + e];
    __syncthreads();
    trsv_lower_f64<float>(r.n, r.S, r.n, ytc);
    double part = 0.0;
    for (int e = threadIdx.x; e < r.n; e += kThreads) part += ytc[e] * ytc[e];
    const double yy = cta_sum(part, sm);
    if (threadIdx.x == 0) t.dchild[r.c] = yy + *r.ld;
}

static int launch_heavy32(const Geom& g, const DevTree<float>& t, const Fork& fk) {
    const size_t sb = sizeof(LaSmem<float>);
    cudaStream_t st = fk.side;
    const long Lr = (long)t.L * t.r;
    const int nmax = fk.heavy_n[0], xt = (int)((Lr + 63) / 64), cv = (int)((Lr + 255) / 256);
    k_heavy32_sigma<<<(unsigned)t.n_heavy_tiles, kThreads, sb, st>>>(g, t);
    int launches = 2;
    long act = t.n_heavy;
    for (int b = 0; 16 * b < nmax; ++b) {
        while (act > 0 && fk.heavy_n[act - 1] <= 16 * b) --act;
        const int rest = nmax - 16 * b - 16 > 0 ? nmax - 16 * b - 16 : 0;
        const int cs = rest > 256 ? (rest + 255) / 256 : 1, ct = b > 0 ? (nmax - 16 * b + 63) / 64 : 0;
        const int tasks = cs + xt * ct;
        k_heavy32_panel<<<(unsigned)(act * tasks), kThreads, sb, st>>>(t, b, cs, ct > 0 ? ct : 1, tasks);
        const int tt = (rest + 63) / 64, tasks2 = cv + tt * (tt + 1) / 2;
        k_heavy32_update<<<(unsigned)(act * tasks2), kThreads, sb, st>>>(t, b, cv, tasks2);
        launches += 2;
    }
    k_heavy32_terms<<<(unsigned)t.n_heavy, kThreads, sb, st>>>(t);
    return launches;
}

// dfin of each sibling group: the sum of its children's terms, in order (the
// slots of regions without observations, and of all but the first of a group
// processed together, stay zero).
template <typename T>
__global__ void k_finest_terms(DevTree<T> t) {
    const long s2 = t.lstart[t.M - 2], cnt2 = level_count(t.J, t.M - 2);
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= cnt2 || skipped(t, s2 + q)) return;
    double s = 0.0;
    for (long c = t.child_lo[q]; c < t.child_hi[q]; ++c) s += t.dchild[c];
    t.dfin[q] = s;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <typename T>
static void launch_cov_set(const Geom& g, const DevTree<T>& t, const CondSetT<T>& s, cudaStream_t st) {
    const long tasks = s.n * t.L;
    const unsigned grid = (unsigned)(tasks < 148L * 32 ? tasks : 148L * 32);
    if constexpr (sizeof(T) == 8)
        with_cov_kind(cov_kind(g, true),
                      [&](auto k) { k_cov_set<T, decltype(k)::value><<<grid, kCovThreads, 0, st>>>(g, t, s); });
    else
        k_cov_set<T, 0><<<grid, kCovThreads, 0, st>>>(g, t, s);
}

template <int RC>
static void launch_condition(const DevTree<double>& t, const CondSet& s, cudaStream_t st) {
    const unsigned grid = (unsigned)s.n;
    if (t.r % 2 == 0) k_condition_set<RC, true><<<grid, kCondThreads, sizeof(CondSmem<RC>), st>>>(t, s);
    else k_condition_set<RC, false><<<grid, kCondThreads, sizeof(CondSmem<RC>), st>>>(t, s);
}

int launch_condition_set(const Geom& g, const DevTree<double>& t, const CondSet& s, cudaStream_t st) {
    launch_cov_set<double>(g, t, s, st);
    if (t.r <= 16) launch_condition<16>(t, s, st);
    else if (t.r <= 32) launch_condition<32>(t, s, st);
    else launch_condition<64>(t, s, st);
    return 2;
}

template <typename T>
int launch_finest(const Geom& g, const DevTree<T>& t, int grid, bool keep, cudaStream_t st, const Fork& fk) {
    int launches = 0;
    if (t.n_chunks > 0) {
        const CondSetT<T> s{t.chunks, t.n_chunks, t.obs0, t.Bhat, t.Ufin, t.sub_lo + t.lstart[t.M - 2],
                            t.sub_hi + t.lstart[t.M - 2]};
        if constexpr (sizeof(T) == 8) {
            if (t.r <= 64) {
                launch_condition_set(g, t, s, st);
            } else {
                launch_cov_set<T>(g, t, s, st);
                k_finest_condition_any<T><<<(unsigned)t.n_chunks, kThreads, sizeof(Tile<64>::Smem), st>>>(t);
            }
        } else {
            launch_cov_set<T>(g, t, s, st);
            k_finest_condition_any<T><<<(unsigned)t.n_chunks, kThreads, sizeof(LaSmem<T>), st>>>(t);
        }
        launches += 2;
    }
    if (t.n_heavy > 0) {
        // the heavy regions' chain of block columns beside the small regions
        cudaEventRecord(fk.fork, st);
        cudaStreamWaitEvent(fk.side, fk.fork, 0);
        if constexpr (sizeof(T) == 4) {
            launches += launch_heavy32(g, t, fk);
        } else {
            const int LT = (int)(((long)t.L * t.r + 63) / 64);
            const size_t sb = sizeof(Tile<64>::Smem);
            with_cov_kind(cov_kind(g, true), [&](auto k) {
                k_cov_heavy<decltype(k)::value><<<(unsigned)t.n_heavy_tiles, kCovThreads, 0, fk.side>>>(g, t);
            });
            k_heavy_sigma<<<(unsigned)t.n_heavy_tiles, kThreads, sb, fk.side>>>(t);
            launches += 2;
            const int nb = (fk.heavy_n[0] + 63) / 64;
            long act = t.n_heavy;
            for (int k = 0; k < nb; ++k) {
                while (act > 0 && fk.heavy_n[act - 1] <= 64 * k) --act;
                const int tiles = k == 0 ? 1 : nb - k + LT;
                k_heavy_column<<<(unsigned)(act * tiles), kThreads, sb, fk.side>>>(t, k, tiles);
                const int below = nb - k - 1 + LT;
                k_heavy_panel<<<(unsigned)(act * below), kThreads, sb, fk.side>>>(t, k, below);
                launches += 2;
            }
        }
        cudaEventRecord(fk.join, fk.side);
    }
    if constexpr (sizeof(T) == 8) {
        launches += launch_finest_small(g, t, keep, st);
    } else if (t.n_fin_items > 0) {
        k_finest_regions_f32<<<(unsigned)(t.n_fin_items < grid ? t.n_fin_items : grid), kThreads, sizeof(LaSmem<T>),
                               st>>>(g, t);
        ++launches;
    }
    if (t.n_heavy > 0) cudaStreamWaitEvent(st, fk.join, 0);
    const long cnt2 = level_count(t.J, t.M - 2);
    k_finest_terms<T><<<(unsigned)((cnt2 + 255) / 256), 256, 0, st>>>(t);
    return launches + 1;
}

cudaError_t prepare_finest() {
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* fn, size_t bytes) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    set((const void*)k_condition_set<16, true>, sizeof(CondSmem<16>));
    set((const void*)k_condition_set<16, false>, sizeof(CondSmem<16>));
    set((const void*)k_condition_set<32, true>, sizeof(CondSmem<32>));
    set((const void*)k_condition_set<32, false>, sizeof(CondSmem<32>));
    set((const void*)k_condition_set<64, true>, sizeof(CondSmem<64>));
    set((const void*)k_condition_set<64, false>, sizeof(CondSmem<64>));
    set((const void*)k_finest_condition_any<double>, sizeof(Tile<64>::Smem));
    set((const void*)k_finest_condition_any<float>, sizeof(LaSmem<float>));
    set((const void*)k_finest_regions_f32, sizeof(LaSmem<float>));
    set((const void*)k_heavy32_sigma, sizeof(LaSmem<float>));
    set((const void*)k_heavy32_panel, sizeof(LaSmem<float>));
    set((const void*)k_heavy32_update, sizeof(LaSmem<float>));
    set((const void*)k_heavy32_terms, sizeof(LaSmem<float>));
    set((const void*)k_heavy_sigma, sizeof(Tile<64>::Smem));
    set((const void*)k_heavy_column, sizeof(Tile<64>::Smem));
    set((const void*)k_heavy_panel, sizeof(Tile<64>::Smem));
    if (e == cudaSuccess) e = prepare_finest_small();
    return e;
}

template int launch_finest<double>(const Geom&, const DevTree<double>&, int, bool, cudaStream_t, const Fork&);
template int launch_finest<float>(const Geom&, const DevTree<float>&, int, bool, cudaStream_t, const Fork&);

}  // namespace mra
