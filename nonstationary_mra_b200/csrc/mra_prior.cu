// Prior of the interior levels (class_approximation.cpp:46-50,84-169): per level,
// the covariance blocks of its regions in one launch, then the regions.
#include "mra_cond.cuh"
#include "mra_tile.cuh"

namespace mra {

// ---------------------------------------------------------------------------
// a2/a3 for the prior: the covariance blocks of one level, in their own launch
// ---------------------------------------------------------------------------
// Regions loc0 .. loc0+nloc-1 (local indices) of level m: block j < m of region
// i is C(Q_{a_j}, Q_i) (rows: the knots of ancestor a_j, columns: the region's
// own knots; evaluate_nonstationary_cross_covariance, evaluate_covariance.cpp:
// 155-234), block m is C(Q_i, Q_i) with sigma^2 + tau^2 on its diagonal
// (:248-313).  Block j of the q-th region goes to out + cov_slot(q, j) r^2,
// column-major with ld r.  One CTA per block at a time; with no barrier-bound
// products beside it the launch keeps every SM full of independent entry
// chains, which the per-region kernel, two CTAs per SM between its products,
// cannot.
// The regions conditioned together (SB siblings) have their blocks of one ancestor
// side by side, as the columns of one r x (SB r) block.
__host__ __device__ inline long cov_slot(long q, int j, int m, int SB) {
    return (q / SB * (m + 1) + j) * SB + q % SB;
}

template <typename T, int KIND>
__global__ void __launch_bounds__(kCovThreads, 4) k_cov_level(Geom g, DevTree<T> t, int m, long loc0, long nloc, int SB,
                                                               T* __restrict__ out) {
    __shared__ __align__(16) double stage[7 * kCovChunk];
    const int r = t.r;
    const long rr = (long)r * r;
    const long s0 = t.lstart[m];
    const long nblocks = nloc * (m + 1);
    for (long b = blockIdx.x; b < nblocks; b += gridDim.x) {
        const long q = (unsigned)b / (unsigned)(m + 1);  // at most 2^31 blocks
        const int j = (int)(b - q * (m + 1));
        const long i = s0 + loc0 + q;
        if (skipped(t, i)) continue;
        const long a = ancestor(t, m, loc0 + q, j);  // the region itself for j == m
        cov_block<T, KIND>(g, t.pts, a * r, r, i * r, r, j == m, out + cov_slot(q, j, m, SB) * rr, r, stage);
    }
}

// Host-side dispatch of the covariance-block launches on the model's form.
template <typename T>
void launch_cov_level(const Geom& g, const DevTree<T>& t, int m, long loc0, long n, int SB, unsigned grid,
                      cudaStream_t st) {
    if constexpr (sizeof(T) == 8)
        with_cov_kind(cov_kind(g, true), [&](auto k) {
            k_cov_level<T, decltype(k)::value><<<grid, kCovThreads, 0, st>>>(g, t, m, loc0, n, SB, t.cbuf);
        });
    else
        k_cov_level<T, 0><<<grid, kCovThreads, 0, st>>>(g, t, m, loc0, n, SB, t.cbuf);
}

// ---------------------------------------------------------------------------
// a5/a6: prior, one level of interior regions
// ---------------------------------------------------------------------------
// The inverse L_a^{-1} of every prior factor is formed once, right after its
// Cholesky, so that the m triangular solves of each descendant become tensor-pipe
// products.  The covariance blocks come from
// k_cov_level (C: the q-th region's m+1 blocks at C + q (m+1) r^2); each
// conditioning product takes its block as the added term, so nothing is
// copied: V_j = C_j - U_{a_j}^T U_{i,0..j-1}, U_{i,j} = L_{a_j}^{-1} V_j and
// K_i = C_i - U_i^T U_i straight into the factor's storage.
//
// FP64, r <= RC <= 64: one CTA per run of SB = min(64 / RC, J) siblings, whose
// ancestors are the same, so that the steps of mra_cond.cuh work on up to 64
// columns whatever r.  Then, per sibling, K_i = C_i - U_i^T U_i from one staged
// operand, lower triangle only, straight into shared memory, where it is factored
// and inverted.  Level of 16,384 regions of 64 knots with 7 ancestors: 14.8 -> 10.7 ms
// (29 TFLOP/s of products, triangles at their own count), of 30 knots: 5.3 -> 1.65 ms,
// against one 256-thread CTA per region with a product routine call per step.
template <int RC, bool EVEN>
__global__ void __launch_bounds__(kCondThreads, CondSmem<RC>::CTAS)
    k_prior_fused(DevTree<double> t, int m, long loc0, long nloc, int SB, const double* __restrict__ C) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using CC = Cond<RC, EVEN>;
    CondSmem<RC>& sm = *reinterpret_cast<CondSmem<RC>*>(la_dyn_smem);
    const int r = t.r;
    const long rr = (long)r * r;
    const long mr = (long)m * r;
    const long q = (long)blockIdx.x * SB;
    const int nsib = (int)(nloc - q < SB ? nloc - q : SB);
    const long i0 = t.lstart[m] + loc0 + q;
    // at the split level of a sharded evaluation siblings belong to different ranks: the columns of a sibling that
    // is not computed here are carried along (columns are independent) and left out below
    bool any = false;
    for (int sib = 0; sib < nsib; ++sib) any = any || !skipped(t, i0 + sib);
    if (!any) return;
    CC cond(sm, r);
    const double* Cq = C + cov_slot(q, 0, m, SB) * rr;
    double* Ui = t.U + t.u_off[m] + (loc0 + q) * mr * r;  // (m r) x (nsib r), ld = m r
    for (int j = 0; j < m; ++j) {
        const long a = ancestor(t, m, loc0 + q, j);
        const CondOp o{t.U + t.u_off[j] + (a - t.lstart[j]) * (long)j * rr, j * r, Ui, mr, nsib * r};
        const double* Cj = Cq + (long)j * SB * rr;
        // the next covariance block (or the self blocks) into L2 while this step's products run
        if (threadIdx.x == 0) prefetch_l2(Cj + (long)SB * rr, (unsigned long)nsib * rr * sizeof(double));
        cond.step(o, t.Pinv + a * rr, Cj, r, nullptr, Ui + (long)j * r);
    }
    for (int sib = 0; sib < nsib; ++sib) {
        if (skipped(t, i0 + sib)) continue;
        const double* Us = Ui + (long)sib * r * mr;
        double acc[2][CC::NF][2];
        const int ns = (int)((mr + TK64 - 1) / TK64);
        auto issue = [&](int v) {  // one operand serves as both factors of U_i^T U_i
            if (v < ns) cond.load_rows(sm.B[v & 1], Us, mr, r, RC, v * TK64, mr);
            cp_async_commit();
        };
        // column fragments up to this warp's rows
        const int nf = 16 * cond.wr < r ? cond.frags(16 * (cond.wr + 1) < r ? 16 * (cond.wr + 1) : r) : 0;
        issue(0);
        cond.init(acc, Cq + ((long)m * SB + sib) * rr, r, r);
        for (int i = 0; i < ns; ++i) {
            cp_async_wait<0>();
            __syncthreads();
            issue(i + 1);
            cond.mma_slab_n(nf, acc, sm.B[i & 1], sm.B[i & 1]);
        }
        double* S = &sm.A[0][0];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int row = 16 * cond.wr + 8 * e + cond.g;
#pragma unroll
            for (int f = 0; f < CC::NF; ++f) {
                const int c = (f * CC::CW + cond.wc) * 8 + 2 * cond.t;
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (c + h < RC)
                        S[row + (c + h) * SLD] = (row < r && c + h < r) ? acc[e][f][h] : (row == c + h ? 1.0 : 0.0);
            }
        }
        __syncthreads();
        const long i = i0 + sib;
        double ld = 0.0;
        const int info =
            potrf_finish<true, CondSmem<RC>, kCondThreads>(r, t.Lprior + i * rr, r, &ld, t.Pinv + i * rr, r);
        if (threadIdx.x == 0) {
            t.ldprior[i] = ld;
            if (info) report_error(t.err, i);
        }
    }
}

// r > 64 (FP64): a region's columns condition on the ancestors in runs of CW columns,
// one CTA each, so that the top levels' few regions still spread over the chip; then
// K_i's lower tiles; then the factors (levels of 1 to 64 regions of 100 knots: 120 to
// 380 us each with one CTA per region doing all of it, 50 to 230 now).
__global__ void __launch_bounds__(kThreads, 2) k_prior_columns(DevTree<double> t, int m, long loc0, long nloc, int CW,
                                                               const double* __restrict__ C) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    Tile<64>::Smem& sm = *reinterpret_cast<Tile<64>::Smem*>(la_dyn_smem);
    const int r = t.r, nc = (r + CW - 1) / CW;
    const long rr = (long)r * r, mr = (long)m * r;
    double* V = t.ws + blockIdx.x * t.ws_stride;  // r x CW
    for (long b = blockIdx.x; b < nloc * nc; b += gridDim.x) {
        const long q = b / nc;
        const int c0 = (int)(b - q * nc) * CW, N = min(CW, r - c0);
        if (skipped(t, t.lstart[m] + loc0 + q)) continue;
        const double* Cq = C + cov_slot(q, 0, m, 1) * rr;
        double* Ui = t.U + t.u_off[m] + (loc0 + q) * mr * r + (long)c0 * mr;
        for (int j = 0; j < m; ++j) {
            const long a = ancestor(t, m, loc0 + q, j);
            cond_tiles(sm, r, t.U + t.u_off[j] + (a - t.lstart[j]) * (long)j * rr, j * r, Ui, mr, N, t.Pinv + a * rr,
                       Cq + j * rr + (long)c0 * r, r, V, r, Ui + (long)j * r);
        }
    }
}

// K_i = C_i - U_i^T U_i, lower tiles, into the factor's storage.
__global__ void __launch_bounds__(kThreads, 2) k_prior_self(DevTree<double> t, int m, long loc0, int nt,
                                                            const double* __restrict__ C) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using TT = Tile<64>;
    TT::Smem& sm = *reinterpret_cast<TT::Smem*>(la_dyn_smem);
    const int r = t.r, tiles = nt * (nt + 1) / 2;
    const long rr = (long)r * r, mr = (long)m * r;
    const long q = blockIdx.x / tiles;
    int s = (int)(blockIdx.x - q * tiles), ti = 0;
    while (s > ti) s -= ++ti;
    const long i = t.lstart[m] + loc0 + q;
    if (skipped(t, i)) return;
    const int r0 = 64 * ti, c0 = 64 * s, M = min(64, r - r0), N = min(64, r - c0);
    const double* Ui = t.U + t.u_off[m] + (loc0 + q) * mr * r;
    const bool vec = r % 2 == 0;
    TT::Acc acc;
    TT::zero(acc);
    TT::add(acc, -1.0, C + cov_slot(q, m, m, 1) * rr + r0 + (long)c0 * r, r, M, N);
    TT::product<true, true>(acc, sm, Ui + r0 * mr, mr, M, Ui + c0 * mr, mr, N, (int)mr, vec, vec);
    TT::store(acc, -1.0, t.Lprior + i * rr + r0 + (long)c0 * r, r, M, N);
}

// r > 128: blocked factorization, the inverse by triangular solves.
__global__ void __launch_bounds__(kThreads, 2) k_prior_factor_any(DevTree<double> t, int m, long loc0) {
    LaSmem<double>& sm = la_smem<double>();
    const long i = t.lstart[m] + loc0 + blockIdx.x, rr = (long)t.r * t.r;
    if (skipped(t, i)) return;
    double ld = 0.0;
    const int info = potrf_lower<double>(t.r, t.Lprior + i * rr, t.r, sm, &ld, t.Pinv + i * rr, t.r);
    if (threadIdx.x == 0) {
        t.ldprior[i] = ld;
        if (info) report_error(t.err, i);
    }
}

// FP32 storage: one CTA per region through the general products.
__global__ void __launch_bounds__(kThreads, 2) k_prior_level_f32(DevTree<float> t, int m, long loc0, long nloc,
                                                                 const float* __restrict__ C) {
    using T = float;
    LaSmem<T>& sm = la_smem<T>();
    const int r = t.r;
    const long rr = (long)r * r;
    const long s0 = level_start(t.J, m);
    const long mr = (long)m * r;
    for (long q = blockIdx.x; q < nloc; q += gridDim.x) {
        const long loc = loc0 + q;
        const long i = s0 + loc;
        if (skipped(t, i)) continue;
        long anc[kMaxLevels];
        {
            long c = i;
            for (int a = m - 1; a >= 0; --a) {
                c = (c - 1) / t.J;
                anc[a] = c;
            }
        }
        const T* Cq = C + cov_slot(q, 0, m, 1) * rr;
        T* Ui = t.U + t.u_off[m] + loc * mr * r;  // (m r) x r, ld = m r
        // one r x r scratch per CTA (stays in L2)
        T* V = t.ws + blockIdx.x * t.ws_stride;
        for (int j = 0; j < m; ++j) {
            const long a = anc[j];
            const T* Cj = Cq + j * rr;
            const T* Vj = Cj;  // level 0 has nothing to condition on
            // the next covariance block (or the self block) into L2 while this step's products run
            if (threadIdx.x == 0) prefetch_l2(Cj + rr, rr * sizeof(T));
            if (j > 0) {
                const T* Ua = t.U + t.u_off[j] + (a - level_start(t.J, j)) * (long)j * rr;
                gemm<T, true, false>(r, r, j * r, (T)-1, Ua, (long)j * r, Ui, mr, (T)1, V, r, sm, Cj, r);
                Vj = V;
            }
            // U_{i,j} = L_a^{-1} V as a product with the stored inverse
            gemm<T, false, false>(r, r, r, (T)1, t.Pinv + a * rr, r, Vj, r, (T)0, Ui + (long)j * r, mr, sm);
        }
        T* Li = t.Lprior + i * rr;
        // K_i = C_i - U_i^T U_i (for m == 0 a product with K = 0: the copy of C_i)
        gemm<T, true, false>(r, r, (int)mr, (T)-1, Ui, mr, Ui, mr, (T)1, Li, r, sm, Cq + (long)m * rr, r);
        double ld = 0.0;
        int info = potrf_lower<T>(r, Li, r, sm, &ld, t.Pinv + i * rr, r);
        if (threadIdx.x == 0) {
            t.ldprior[i] = ld;
            if (info) report_error(t.err, i);
        }
    }
}

// The factors of a level's regions, 64 < r <= 128.
__global__ void __launch_bounds__(kThreads, 1) k_prior_factor(DevTree<double> t, int m, long loc0) {
    const long i = t.lstart[m] + loc0 + blockIdx.x, rr = (long)t.r * t.r;
    if (skipped(t, i)) return;
    double ld = 0.0;
    const int info = potrf_128(t.r, t.Lprior + i * rr, t.r, &ld, t.Pinv + i * rr, t.r);
    if (threadIdx.x == 0) {
        t.ldprior[i] = ld;
        if (info) report_error(t.err, i);
    }
}

// ---------------------------------------------------------------------------
// launcher
// ---------------------------------------------------------------------------
template <int RC>
static void launch_fused(const DevTree<double>& t, int m, long loc0, long n, int SB, unsigned runs, cudaStream_t st) {
    if (t.r % 2 == 0)
        k_prior_fused<RC, true><<<runs, kCondThreads, sizeof(CondSmem<RC>), st>>>(t, m, loc0, n, SB, t.cbuf);
    else
        k_prior_fused<RC, false><<<runs, kCondThreads, sizeof(CondSmem<RC>), st>>>(t, m, loc0, n, SB, t.cbuf);
}

template <typename T>
int launch_prior_level(const Geom& g, const DevTree<T>& t, int m, int grid, cudaStream_t st, CovTiming* tm) {
    auto mark = [&](cudaEvent_t e) {
        if (tm->capturing) cudaEventRecordWithFlags(e, st, cudaEventRecordExternal);
        else cudaEventRecord(e, st);
    };
    const long cnt = level_count(t.J, m);
    const int SB = prior_batch(sizeof(T) == 8, t.r, t.J);
    const long per_region = (long)(m + 1) * t.r * t.r;
    long per = t.cbuf_elems / (per_region * SB) * SB;  // regions whose blocks fit the buffer at once
    int launches = 0;
    for (long loc0 = 0; loc0 < cnt; loc0 += per) {
        const long n = cnt - loc0 < per ? cnt - loc0 : per;
        const long nb = n * (m + 1);
        const long cov_grid = (long)grid * 16;  // 16 per region-kernel slot: 32 CTAs per SM
        const bool timed = tm && tm->used < tm->cap;
        if (tm && !timed) tm->overflow = true;
        if (timed) mark(tm->ev[2 * tm->used]);
        launch_cov_level<T>(g, t, m, loc0, n, SB, (unsigned)(nb < cov_grid ? nb : cov_grid), st);
        if (timed) mark(tm->ev[2 * tm->used++ + 1]);
        if constexpr (sizeof(T) == 4) {
            k_prior_level_f32<<<(unsigned)(n < grid ? n : grid), kThreads, sizeof(LaSmem<T>), st>>>(t, m, loc0, n, t.cbuf);
        } else if (t.r <= 64) {
            const unsigned runs = (unsigned)((n + SB - 1) / SB);
            if (t.r <= 16) launch_fused<16>(t, m, loc0, n, SB, runs, st);
            else if (t.r <= 32) launch_fused<32>(t, m, loc0, n, SB, runs, st);
            else launch_fused<64>(t, m, loc0, n, SB, runs, st);
        } else {
            const size_t sb = sizeof(Tile<64>::Smem);
            if (m > 0) {
                int CW = 64;  // narrower runs while there are fewer than CTAs
                while (CW > 16 && n * ((t.r + CW - 1) / CW) < grid) CW /= 2;
                const long items = n * ((t.r + CW - 1) / CW);
                k_prior_columns<<<(unsigned)(items < grid ? items : grid), kThreads, sb, st>>>(t, m, loc0, n, CW, t.cbuf);
                ++launches;
            }
            const int nt = (t.r + 63) / 64;
            k_prior_self<<<(unsigned)(n * (nt * (nt + 1) / 2)), kThreads, sb, st>>>(t, m, loc0, nt, t.cbuf);
            if (t.r <= 128) k_prior_factor<<<(unsigned)n, kThreads, sizeof(Potrf128Smem), st>>>(t, m, loc0);
            else k_prior_factor_any<<<(unsigned)n, kThreads, sizeof(LaSmem<double>), st>>>(t, m, loc0);
            ++launches;
        }
        launches += 2;
    }
    return launches;
}

cudaError_t prepare_prior() {
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* fn, size_t bytes) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    set((const void*)k_prior_factor, sizeof(Potrf128Smem));
    set((const void*)k_prior_columns, sizeof(Tile<64>::Smem));
    set((const void*)k_prior_self, sizeof(Tile<64>::Smem));
    set((const void*)k_prior_factor_any, sizeof(LaSmem<double>));
    set((const void*)k_prior_level_f32, sizeof(LaSmem<float>));
    set((const void*)k_prior_fused<16, true>, sizeof(CondSmem<16>));
    set((const void*)k_prior_fused<16, false>, sizeof(CondSmem<16>));
    set((const void*)k_prior_fused<32, true>, sizeof(CondSmem<32>));
    set((const void*)k_prior_fused<32, false>, sizeof(CondSmem<32>));
    set((const void*)k_prior_fused<64, true>, sizeof(CondSmem<64>));
    set((const void*)k_prior_fused<64, false>, sizeof(CondSmem<64>));
    return e;
}

cudaError_t set_gemm_tiles_prior(const int nw[3]) { return cudaMemcpyToSymbol(c_gemm_nw, nw, 3 * sizeof(int)); }

template int launch_prior_level<double>(const Geom&, const DevTree<double>&, int, int, cudaStream_t, CovTiming*);
template int launch_prior_level<float>(const Geom&, const DevTree<float>&, int, int, cudaStream_t, CovTiming*);

}  // namespace mra
