// Region kernels of the MRA hot path, templated on the storage type T
// (double: plain FP64 path; float: mixed path, FP32 storage and 3xTF32 tensor
// products, FP64 diagonal blocks and log-likelihood accumulation).
//
// Schedule of one log-likelihood (one launch per stage and tree level):
//   k_fields            sigma^2/beta/tau^2 at every knot, observation and
//                       prediction point (class_nonstationary_covariance.cpp:479-573)
//   k_prior_level(m)    levels 0..M-2, one CTA per region: U_{i,j} = L_{a_j}^{-1} V_j,
//                       L_i = chol(K_i)   (class_approximation.cpp:46-50,84-169)
//   (mra_finest.cu)     finest level: conditioning, Sigma, L_Sigma, y~, B^ and
//                       the log-lik terms
//                       (...-loop-regions-at-finest-level-in-prior.cpp:90-269)
//   k_posterior_level(m) levels M-2..0 (...-posterior-inference.cpp:14-265,
//                       class_approximation.cpp:186-306)
//   k_reduce            deterministic sum of the per-region terms
//   k_predict           prediction, one CTA per level M-2 region (its finest
//                       children's predictions together)
//                       (...-prior.cpp:271-392, class_approximation-predict.cpp:105-189)
//
// Posterior representation.  A region's contribution to its parent is the pair
// (A~, w~) of the reference (class_approximation.cpp:266-306).  Below a size
// threshold it is carried in factored observation-space form instead: a matrix
// F (n x m r, one row per observation of the subtree) and a vector f with
// A~_(j,k) = F_j^T F_k and w~_j = F_j^T f.  The finest level starts in this
// form (F = B^, f = y~).  For a region i at level m with factored input (F, f):
//   Y = L_i^{-1} F_m^T,  R R^T = I + Y^T Y,
//   output F' = R^{-1} F_{0..m-1},  f' = R^{-1} f,
//   log-lik term 2 log|R| - (f^T f - f'^T f'),
// which equals the reference's -2 log|L_i| + 2 log|L~_i| - v^T v with
// L~ L~^T = L L^T + F_m^T F_m (Sylvester's determinant identity and Woodbury),
// and F'^T F' / F'^T f' equal the reference's A~ / w~ of the region.  Larger
// regions use the reference's dense r x r slices.  Prediction mode also forms
// L~, v and G of factored regions from (F, f).
#include "mra_kernels.cuh"

namespace mra {

// ---------------------------------------------------------------------------
// a1: fields
// ---------------------------------------------------------------------------
__global__ void k_fields(Geom g, FieldParams fp, const double* __restrict__ c0, const double* __restrict__ c1,
                         const double* __restrict__ c2, long n, double* __restrict__ s2, double* __restrict__ beta,
                         double* __restrict__ t2) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* th = fp.theta;
    if (!g.nonstat) {
        s2[i] = th[6];
        beta[i] = th[7];
        t2[i] = th[8];
        return;
    }
    Pt p{c0[i], c1[i], c2[i]};
    double out[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        double v = th[3 + f];
        const long nb = fp.nb[f];
        const double* c = fp.centers[f];
        const double* w = fp.weights[f];
        for (long b = 0; b < nb; ++b) {
            Pt q{c[b], c[nb + b], c[2 * nb + b]};
            double d = point_distance(g, p, q) / fp.basis_len;
            if (fp.basis == 0) {
                if (d >= 1) continue;
                double u = 1 - d, u2 = u * u;
                v += u2 * u2 * u2 * (35 * d * d + 18 * d + 3) * w[b] / 3;
            } else {
                v += exp(-0.5 * d * d) * w[b];
            }
        }
        out[f] = th[f] * exp(v);
    }
    s2[i] = out[0];
    beta[i] = out[1];
    t2[i] = out[2];
}

// ---------------------------------------------------------------------------
// a2/a3 for the prior: the covariance blocks of one level, in their own launch
// ---------------------------------------------------------------------------
// Regions loc0 .. loc0+nloc-1 (local indices) of level m: block j < m of region
// i is C(Q_{a_j}, Q_i) (rows: the knots of ancestor a_j, columns: the region's
// own knots; evaluate_nonstationary_cross_covariance, evaluate_covariance.cpp:
// 155-234), block m is C(Q_i, Q_i) with sigma^2 + tau^2 on its diagonal
// (:248-313).  Block j of the q-th region goes to out + (q (m+1) + j) r^2,
// column-major with ld r.  One CTA per block at a time; with no barrier-bound
// products beside it the launch keeps every SM full of independent entry
// chains, which the per-region kernel, two CTAs per SM between its products,
// cannot.
template <typename T, int KIND>
__global__ void __launch_bounds__(kCovThreads, 4) k_cov_level(Geom g, DevTree<T> t, int m, long loc0, long nloc,
                                                               T* __restrict__ out) {
    __shared__ double stage[7 * kCovChunk];
    const int r = t.r;
    const long rr = (long)r * r;
    const long s0 = level_start(t.J, m);
    const long nblocks = nloc * (m + 1);
    for (long b = blockIdx.x; b < nblocks; b += gridDim.x) {
        const long q = b / (m + 1);
        const int j = (int)(b - q * (m + 1));
        const long i = s0 + loc0 + q;
        if (skipped(t, i)) continue;
        long a = i;  // the ancestor of level j (the region itself for j == m)
        for (int l = m; l > j; --l) a = (a - 1) / t.J;
        cov_block<T, KIND>(g, t.pts, a * r, r, i * r, r, j == m, out + b * rr, r, stage);
    }
}

// Host-side dispatch of the covariance-block launches on the model's form.
template <typename T>
void launch_cov_level(const Geom& g, const DevTree<T>& t, int m, long loc0, long n, unsigned grid, cudaStream_t st) {
    switch (cov_kind(g, sizeof(T) == 8)) {
        case 1: k_cov_level<T, 1><<<grid, kCovThreads, 0, st>>>(g, t, m, loc0, n, t.cbuf); break;
        case 2: k_cov_level<T, 2><<<grid, kCovThreads, 0, st>>>(g, t, m, loc0, n, t.cbuf); break;
        case 3: k_cov_level<T, 3><<<grid, kCovThreads, 0, st>>>(g, t, m, loc0, n, t.cbuf); break;
        case 4: k_cov_level<T, 4><<<grid, kCovThreads, 0, st>>>(g, t, m, loc0, n, t.cbuf); break;
        default: k_cov_level<T, 0><<<grid, kCovThreads, 0, st>>>(g, t, m, loc0, n, t.cbuf); break;
    }
}

// ---------------------------------------------------------------------------
// a5/a6: prior, one level of interior regions
// ---------------------------------------------------------------------------
// One CTA per region.  The inverse L_a^{-1} of every prior factor is formed
// once, right after its Cholesky, so that the m triangular solves of each
// descendant become tensor-pipe products.  The covariance blocks come from
// k_cov_level (C: the q-th region's m+1 blocks at C + q (m+1) r^2); each
// conditioning product takes its block as the added term, so nothing is
// copied: V_j = C_j - U_{a_j}^T U_{i,0..j-1}, U_{i,j} = L_{a_j}^{-1} V_j and
// K_i = C_i - U_i^T U_i straight into the factor's storage.
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_prior_level(Geom g, DevTree<T> t, int m, long loc0, long nloc,
                                                            const T* __restrict__ C) {
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
        const T* Cq = C + q * (long)(m + 1) * rr;
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
                gemm_wide<T, true, false>(r, r, j * r, (T)-1, Ua, (long)j * r, Ui, mr, (T)1, V, r, sm, Cj, r);
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

// ---------------------------------------------------------------------------
// posterior steps of one region (level m): factored and dense forms
// ---------------------------------------------------------------------------
// The products of the posterior steps go through a separate function: the
// steps keep many values live across their products, and inlined there the
// product loops would share (and spill) their registers.
template <typename T, bool TA, bool TB, bool ONE_TILE = false>
__device__ __noinline__ void gemm_call(int M, int N, int K, T alpha, const T* A, long lda, const T* B, long ldb,
                                       T beta, T* C, long ldc, LaSmem<T>& sm, const T* Cin = nullptr,
                                       long ldcin = 0) {
    gemm<T, TA, TB, ONE_TILE>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, sm, Cin, ldcin);
}

// Factored input (F: n rows of width (m+1) r, row stride ldF; f: n doubles).
// Writes F' (n rows of width m r) to Fo and f' to fo when m > 0.
template <typename T>
__device__ __noinline__ void factored_step(const DevTree<T>& t, int m, long i, int n, const T* F, long ldF, const double* f, T* Fo,
                              double* fo, bool keep, T* ws, double* wsd, LaSmem<T>& sm, double& dterm) {
    const int r = t.r;
    const long rr = (long)r * r, mr = (long)m * r;
    const T* Li = t.Lprior + i * rr;
    T* Y = ws;                  // r x n
    T* S = ws + (long)r * n;    // n x n
    T* Rinv = S + (long)n * n;  // n x n (n <= 128)
    // Y = L_i^{-1} F_m^T as a product with the stored inverse of the prior factor
    gemm_call<T, false, false>(r, n, r, (T)1, t.Pinv + i * rr, r, F + mr, ldF, (T)0, Y, r, sm);
    gemm_call<T, true, false>(n, n, r, (T)1, Y, r, Y, r, (T)0, S, n, sm);
    for (int q = threadIdx.x; q < n; q += kThreads) S[q + (long)q * n] += (T)1;
    __syncthreads();
    double ld = 0.0;
    const bool small = sizeof(T) == 8 && n <= 128;
    int info = potrf_lower<T>(n, S, n, sm, &ld, small ? Rinv : nullptr, n);
    double* fp = m > 0 ? fo : wsd;
    double part = 0.0;
    for (int q = threadIdx.x; q < n; q += kThreads) {
        fp[q] = f[q];
        part += f[q] * f[q];
    }
    double ff = cta_sum(part, sm);
    if (small) trmv_lower_inv<T>(n, Rinv, n, fp, fp);  // f' = R^{-1} f with the inverse formed above
    else trsv_lower_f64<T>(n, S, n, fp);
    part = 0.0;
    for (int q = threadIdx.x; q < n; q += kThreads) part += fp[q] * fp[q];
    double pp = cta_sum(part, sm);
    if (threadIdx.x == 0) {
        dterm += ld - (ff - pp);
        if (info) report_error(t.err, i);
    }
    if (m > 0) {
        if (small) {
            // F' = F_{0..m-1} R^{-T}
            gemm_call<T, false, true>((int)mr, n, n, (T)1, F, ldF, Rinv, n, (T)0, Fo, mr, sm);
        } else {
            for (long e = threadIdx.x; e < mr * n; e += kThreads) {
                long x = e % mr, q = e / mr;
                Fo[q * mr + x] = F[q * ldF + x];
            }
            __syncthreads();
            trsm_right_lower_trans<T>((int)mr, n, S, n, Fo, mr, sm);
        }
    }
    if (keep) {
        // predictive factors of the region: L~ L~^T = L L^T + F_m^T F_m, v = L~^{-1} F_m^T f,
        // G = L~^{-1} F_m^T F_{0..m-1}
        T* Lt = t.Lpost + i * rr;
        gemm_call<T, false, true>(r, r, r, (T)1, Li, r, Li, r, (T)0, Lt, r, sm);
        gemm_call<T, false, true>(r, r, n, (T)1, F + mr, ldF, F + mr, ldF, (T)1, Lt, r, sm);
        T* Lti = t.Lpinv ? t.Lpinv + i * rr : nullptr;  // L~^{-1}, kept for prediction
        int info2 = potrf_lower<T>(r, Lt, r, sm, nullptr, Lti, r);
        double* v = t.vpost + i * r;
        for (int tt = threadIdx.x; tt < r; tt += kThreads) {
            double s = 0.0;
            for (int q = 0; q < n; ++q) s += (double)F[(long)q * ldF + mr + tt] * f[q];
            v[tt] = s;
        }
        __syncthreads();
        if (Lti) trmv_lower_inv<T>(r, Lti, r, v, v);
        else trsv_lower_f64<T>(r, Lt, r, v);
        if (m > 0) {
            T* Gi = t.G + t.u_off[m] + (i - level_start(t.J, m)) * mr * r;
            gemm_call<T, false, true>(r, (int)mr, n, (T)1, F + mr, ldF, F, ldF, (T)0, Gi, r, sm);
            // G = L~^{-1} G in place: one row tile (r <= 64) reads all of its
            // column block before writing it
            if (Lti) gemm_call<T, false, false>(r, (int)mr, r, (T)1, Lti, r, Gi, r, (T)0, Gi, r, sm);
            else trsm_left_lower<T>(r, (int)mr, Lt, r, Gi, r, sm);
        }
        if (info2 && threadIdx.x == 0) report_error(t.err, i);
    }
}

// Dense input: Aagg holds the slices (j,k), j <= k <= m, of the summed children
// contributions, wagg the (m+1) x r summed w.
template <typename T>
__device__ __noinline__ void dense_step(const DevTree<T>& t, int m, long i, const T* Aagg, const double* wagg, bool keep, T* Gw,
                           LaSmem<T>& sm, double& dterm) {
    const int r = t.r;
    const long rr = (long)r * r, mr = (long)m * r;
    const long loc = i - level_start(t.J, m);
    const T* Lp = t.Lprior + i * rr;
    T* Lt = t.Lpost + i * rr;
    gemm_call<T, false, true>(r, r, r, (T)1, Lp, r, Lp, r, (T)0, Lt, r, sm);
    const T* Amm = Aagg + slice_index(m + 1, m, m) * rr;
    for (long e = threadIdx.x; e < rr; e += kThreads) Lt[e] += Amm[e];
    __syncthreads();
    double ld = 0.0;
    // L~^{-1}: kept for prediction when that is on, else an r x r scratch after the G scratch
    const bool kept = keep && t.Lpinv;
    T* Ltinv = kept ? t.Lpinv + i * rr : Gw + mr * r;
    const bool small = sizeof(T) == 8 && r <= 64 && (m > 0 || kept);
    int info = potrf_lower<T>(r, Lt, r, sm, &ld, small ? Ltinv : nullptr, r);
    double* v = t.vpost + i * r;
    for (int e = threadIdx.x; e < r; e += kThreads) v[e] = wagg[mr + e];
    __syncthreads();
    if (small) trmv_lower_inv<T>(r, Ltinv, r, v, v);  // v = L~^{-1} w_m with the inverse formed above
    else trsv_lower_f64<T>(r, Lt, r, v);
    double part = 0.0;
    for (int e = threadIdx.x; e < r; e += kThreads) part += v[e] * v[e];
    double vv = cta_sum(part, sm);
    if (threadIdx.x == 0) {
        dterm += ld - t.ldprior[i] - vv;
        if (info) report_error(t.err, i);
    }
    if (m == 0) return;
    T* Gi = keep ? t.G + t.u_off[m] + loc * mr * r : Gw;  // r x (m r), ld = r
    if (small) {
        // G_j = L~^{-1} A_(j,m)^T
        for (int j = 0; j < m; ++j)
            gemm_call<T, false, true>(r, r, r, (T)1, Ltinv, r, Aagg + slice_index(m + 1, j, m) * rr, r, (T)0,
                                 Gi + (long)j * rr, r, sm);
    } else {
        for (long e = threadIdx.x; e < mr * r; e += kThreads) {
            int j = (int)(e / rr);
            long w = e % rr;
            int p = (int)(w % r), q = (int)(w / r);
            Gi[e] = Aagg[slice_index(m + 1, j, m) * rr + q + (long)p * r];  // G_j = A_(j,m)^T
        }
        __syncthreads();
        trsm_left_lower<T>(r, (int)mr, Lt, r, Gi, r, sm);
    }
    const long slot = t.dslot[i];  // compact index among the level's dense regions
    double* wo = t.wout[m & 1] + slot * mr;
    for (long x = threadIdx.x; x < mr; x += kThreads) {
        double s = 0.0;
        for (int tt = 0; tt < r; ++tt) s += (double)Gi[tt + x * r] * v[tt];
        wo[x] = wagg[x] - s;
    }
    // A_out(j, j..m-1) = A(j, j..m-1) - G_j^T G_{j..m-1}: both slice rows are
    // contiguous r x r blocks, one product per j reading A from Aagg
    T* ao = t.aout[m & 1] + slot * n_slices(m) * rr;
    for (int j = 0; j < m; ++j) {
        T* dst = ao + slice_index(m, j, j) * rr;
        const T* src = Aagg + slice_index(m + 1, j, j) * rr;
        gemm_call<T, true, false>(r, (m - j) * r, r, (T)-1, Gi + (long)j * rr, r, Gi + (long)j * rr, r, (T)1, dst, r,
                                  sm, src, r);
    }
}

// Aagg/wagg += the (A~, w~) of factored rows F (n x (m+1) r, row stride ldF), f;
// with `init` they are set instead (the first contribution: no zeroing pass).
// The slices (j, j..m) of A~ are contiguous r x r blocks, so block row j is
// one product F_j^T F_{j..m} (r x (m+1-j) r).
template <typename T>
__device__ __noinline__ void accumulate_factored(const DevTree<T>& t, int m, int n, const T* F, long ldF, const double* f, T* Aagg,
                                    double* wagg, bool init, LaSmem<T>& sm) {
    const int r = t.r;
    const long rr = (long)r * r, mr1 = (long)(m + 1) * r;
    if (n == 0) {
        if (init) {
            for (long e = threadIdx.x; e < n_slices(m + 1) * rr; e += kThreads) Aagg[e] = (T)0;
            for (long e = threadIdx.x; e < mr1; e += kThreads) wagg[e] = 0.0;
            __syncthreads();
        }
        return;
    }
    for (int j = 0; j <= m; ++j)
        gemm_call<T, false, true>(r, (m + 1 - j) * r, n, (T)1, F + (long)j * r, ldF, F + (long)j * r, ldF,
                                  init ? (T)0 : (T)1, Aagg + slice_index(m + 1, j, j) * rr, r, sm);
    for (long x = threadIdx.x; x < mr1; x += kThreads) {
        double s = 0.0;
        for (int q = 0; q < n; ++q) s += (double)F[(long)q * ldF + x] * f[q];
        wagg[x] = init ? s : wagg[x] + s;
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// a9/a10/a11: posterior, one level (m = M-3 .. 0)
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_posterior_level(Geom g, DevTree<T> t, int m, int keep) {
    LaSmem<T>& sm = la_smem<T>();
    const int r = t.r;
    const long rr = (long)r * r, mr1 = (long)(m + 1) * r;
    const long s0 = level_start(t.J, m), cnt = level_count(t.J, m);
    const long ns_in = n_slices(m + 1);
    T* ws = t.ws + blockIdx.x * t.ws_stride;
    double* wsd = t.wsd + blockIdx.x * t.wsd_stride;
    const T* Fin = t.Fbuf[(m + 1) & 1];
    const double* fin = t.fbuf[(m + 1) & 1];
    const T* ain = t.aout[(m + 1) & 1];
    const double* win = t.wout[(m + 1) & 1];
    const bool from_finest = m == t.M - 2;  // children are finest regions: rows of B^, y~
    // regions taken from a shared counter, most expensive first (the clustered
    // regions' dense steps cost tens of factored ones)
    __shared__ long s_loc;
    for (;;) {
        __syncthreads();  // every thread has read the previous s_loc
        if (threadIdx.x == 0) {
            const int q = atomicAdd(&t.queue[kQueuePost + m], 1);
            s_loc = q < cnt ? t.post_order[s0 + q] : -1;
        }
        __syncthreads();
        const long loc = s_loc;
        if (loc < 0) break;
        const long i = s0 + loc;
        if (skipped(t, i)) continue;
        double dterm = 0.0;
        if (from_finest) {
            const long lo = t.sub_lo[i];
            const int n = (int)(t.sub_hi[i] - lo);
            const T* F = t.Bhat + lo * mr1;
            const double* f = t.yt + lo;
            if (t.factored[i]) {
                T* Fo = m > 0 ? t.Fbuf[m & 1] + lo * (long)m * r : nullptr;
                double* fo = m > 0 ? t.fbuf[m & 1] + lo : nullptr;
                factored_step<T>(t, m, i, n, F, mr1, f, Fo, fo, keep != 0, ws, wsd, sm, dterm);
            } else {
                T* Aagg = ws;
                double* wagg = wsd;
                accumulate_factored<T>(t, m, n, F, mr1, f, Aagg, wagg, true, sm);
                dense_step<T>(t, m, i, Aagg, wagg, keep != 0, Aagg + ns_in * rr, sm, dterm);
            }
        } else if (t.factored[i]) {
            const long lo = t.sub_lo[i];
            const int n = (int)(t.sub_hi[i] - lo);
            T* Fo = m > 0 ? t.Fbuf[m & 1] + lo * (long)m * r : nullptr;
            double* fo = m > 0 ? t.fbuf[m & 1] + lo : nullptr;
            factored_step<T>(t, m, i, n, Fin + lo * mr1, mr1, fin + lo, Fo, fo, keep != 0, ws, wsd, sm, dterm);
        } else {
            T* Aagg = ws;
            double* wagg = wsd;
            bool first = true;  // the first contribution sets Aagg / wagg
            for (int cc = 1; cc <= t.J; ++cc) {
                const long c = i * t.J + cc;
                if (t.factored[c]) {
                    // factored children with adjacent rows are accumulated together
                    const long lo = t.sub_lo[c];
                    long hi = t.sub_hi[c], cl = c;
                    while (cc < t.J && t.factored[cl + 1] && t.sub_lo[cl + 1] == hi) {
                        ++cc;
                        ++cl;
                        hi = t.sub_hi[cl];
                    }
                    accumulate_factored<T>(t, m, (int)(hi - lo), Fin + lo * mr1, mr1, fin + lo, Aagg, wagg, first, sm);
                } else {
                    const long cl = t.dslot[c];
                    const T* as = ain + cl * ns_in * rr;
                    const double* wsrc = win + cl * mr1;
                    for (long e = threadIdx.x; e < ns_in * rr; e += kThreads) Aagg[e] = first ? as[e] : Aagg[e] + as[e];
                    for (long e = threadIdx.x; e < mr1; e += kThreads) wagg[e] = first ? wsrc[e] : wagg[e] + wsrc[e];
                    __syncthreads();
                }
                first = false;
            }
            dense_step<T>(t, m, i, Aagg, wagg, keep != 0, Aagg + ns_in * rr, sm, dterm);
        }
        if (threadIdx.x == 0) t.dpost[i] = dterm;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// a12: prediction
// ---------------------------------------------------------------------------
// For every prediction q < np, one warp forms ss = sum_x c_x^2 and
// mm = sum_x c_x v_x over the column c = C + q ldc (len entries; v may be
// null) with a fixed lane -> entry mapping and shuffle tree, and lane 0 applies
// var[q] += sgn * ss, mean[q] = (add_mean ? mean[q] : 0) + mm.  Ends with a barrier.
template <typename T>
__device__ inline void predict_column_sums(int np, const T* C, long ldc, int len, const double* v, double sgn,
                                           bool add_mean, double* var, double* mean) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int q = w; q < np; q += kThreads / 32) {
        const T* col = C + (long)q * ldc;
        double ss = 0.0, mm = 0.0;
        for (int x = lane; x < len; x += 32) {
            const double c = (double)col[x];
            ss += c * c;
            if (v) mm += c * v[x];
        }
        for (int o = 16; o > 0; o >>= 1) {
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
            mm += __shfl_xor_sync(0xffffffffu, mm, o);
        }
        if (lane == 0) {
            var[q] += sgn * ss;
            if (v) mean[q] = (add_mean ? mean[q] : 0.0) + mm;
        }
    }
    __syncthreads();
}

// One CTA per level M-2 region: the finest children of a region share all of
// their ancestors, so the conditioning of the group's predictions on the
// ancestors (prior part) and the posterior pass back over the ancestors run
// once for all of them; only the part of each finest region's own
// observations runs per child.
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_predict(Geom g, DevTree<T> t) {
    LaSmem<T>& sm = la_smem<T>();
    __shared__ long s_k;
    const int r = t.r, L = t.L;
    const long rr = (long)r * r, Lr = (long)L * r;
    const long cnt2 = level_count(t.J, t.M - 2);
    for (;;) {
        if (threadIdx.x == 0) {
            int q = atomicAdd(&t.queue[1], 1);
            s_k = q < cnt2 ? t.pred_order[q] : -1;
        }
        __syncthreads();
        const long gl = s_k;
        __syncthreads();
        if (gl < 0) break;
        const long clo = t.child_lo[gl], chi = t.child_hi[gl];
        if (chi <= clo) continue;
        const long p0 = t.pred_off[clo];
        const int np = (int)(t.pred_off[chi] - p0);
        if (np == 0) continue;
        const int64_t* anc = t.fin_anc + clo * L;  // shared by every finest child of the region
        T* P = t.P + p0 * Lr;
        T* Bt = t.Bt + p0 * Lr;
        for (int j = 0; j < L; ++j) {
            const long a = anc[j];
            T* Cj = Bt + (long)j * r;
            fill_cov<T>(g, t.pts, a * r, r, t.pred0 + p0, np, false, Cj, Lr, sm);
            __syncthreads();
            if (j > 0) {
                const T* Ua = t.U + t.u_off[j] + (a - level_start(t.J, j)) * (long)j * rr;
                gemm<T, true, false>(r, np, j * r, (T)-1, Ua, (long)j * r, P, Lr, (T)1, Cj, Lr, sm);
            }
            // P_j = L_a^{-1} C_j as a product with the stored inverse of the prior factor
            gemm<T, false, false>(r, np, r, (T)1, t.Pinv + a * rr, r, Cj, Lr, (T)0, P + (long)j * r, Lr, sm);
        }
        double* mean = t.mean + p0;
        double* var = t.var + p0;
        for (int q = threadIdx.x; q < np; q += kThreads) {
            const long ip = t.pred0 + p0 + q;
            var[q] = t.pts.s2[ip] + t.pts.t2[ip];
            mean[q] = 0.0;
        }
        __syncthreads();
        predict_column_sums<T>(np, P, Lr, (int)Lr, nullptr, -1.0, false, var, mean);
        for (long k = clo; k < chi; ++k) {
            const long pk = t.pred_off[k];
            const int npk = (int)(t.pred_off[k + 1] - pk);
            const long o0 = t.obs_off[k];
            const int n = (int)(t.obs_off[k + 1] - o0);
            if (npk == 0 || n == 0) continue;
            T* Pk = t.P + pk * Lr;
            T* Pc = t.Pc + t.pc_off[k];  // n x npk, ld = n
            fill_cov<T>(g, t.pts, t.obs0 + o0, n, t.pred0 + pk, npk, false, Pc, n, sm);
            __syncthreads();
            gemm<T, true, false>(n, npk, (int)Lr, (T)-1, t.Ufin + o0 * Lr, Lr, Pk, Lr, (T)1, Pc, n, sm);
            trsm_left_lower<T>(n, npk, t.Lsig + t.lsig_off[k], n, Pc, n, sm);
            predict_column_sums<T>(npk, Pc, n, n, t.yt + o0, -1.0, false, var + (pk - p0), mean + (pk - p0));
            gemm<T, false, false>((int)Lr, npk, n, (T)-1, t.Bhat + o0 * Lr, Lr, Pc, n, (T)1, t.Bt + pk * Lr, Lr, sm);
        }
        for (int j = L - 1; j >= 0; --j) {
            const long a = anc[j];
            T* KcB = Bt + (long)j * r;
            if (t.Lpinv) {
                // L~_a^{-1} KcB in place (one row tile, r <= 64)
                gemm<T, false, false>(r, np, r, (T)1, t.Lpinv + a * rr, r, KcB, Lr, (T)0, KcB, Lr, sm);
            } else {
                trsm_left_lower<T>(r, np, t.Lpost + a * rr, r, KcB, Lr, sm);
            }
            if (j > 0) {
                const T* Ga = t.G + t.u_off[j] + (a - level_start(t.J, j)) * (long)j * rr;
                gemm<T, true, false>(j * r, np, r, (T)-1, Ga, r, KcB, Lr, (T)1, Bt, Lr, sm);
            }
            predict_column_sums<T>(np, KcB, Lr, r, t.vpost + a * r, 1.0, true, var, mean);
        }
    }
}

// ---------------------------------------------------------------------------
// deterministic final sum: d = sum(dpost) + sum(dfin)
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_reduce(DevTree<T> t, double* out) {
    LaSmem<T>& sm = la_smem<T>();
    double s = 0.0;
    for (long i = threadIdx.x; i < t.n_int; i += kThreads) s += t.dpost[i];
    const long cnt2 = level_count(t.J, t.M - 2);
    for (long i = threadIdx.x; i < cnt2; i += kThreads) s += t.dfin[i];
    double tot = cta_sum(s, sm);
    if (threadIdx.x == 0) out[0] = tot;
}

// ---------------------------------------------------------------------------
// prior sample y = sum_j U_{obs,j}^T z_{a_j} + L_Sigma z_obs
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_sample(DevTree<T> t, const double* z_int, const double* z_obs,
                                                    double* y_out) {
    const int r = t.r, L = t.L;
    const long Lr = (long)L * r;
    for (long k = blockIdx.x; k < t.n_fin; k += gridDim.x) {
        const long o0 = t.obs_off[k];
        const int n = (int)(t.obs_off[k + 1] - o0);
        const int64_t* anc = t.fin_anc + k * L;
        const T* S = t.Lsig + t.lsig_off[k];
        for (int q = threadIdx.x; q < n; q += kThreads) {
            const T* col = t.Ufin + (o0 + q) * Lr;
            double y = 0.0;
            for (int j = 0; j < L; ++j) {
                const double* z = z_int + anc[j] * r;
                for (int x = 0; x < r; ++x) y += (double)col[(long)j * r + x] * z[x];
            }
            for (int x = 0; x <= q; ++x) y += (double)S[q + (long)x * n] * z_obs[o0 + x];
            y_out[o0 + q] = y;
        }
    }
}

// ---------------------------------------------------------------------------
// evaluate_*covariance blocks (layout out[i1*n2 + i2])
// ---------------------------------------------------------------------------
__global__ void k_cov_block(Geom g, PointSet P, long a0, int na, long b0, int nb, int self, double* out) {
    long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long)na * nb) return;
    int tt = (int)(e % na), q = (int)(e / na);
    long ia = a0 + tt, ib = b0 + q;
    double v;
    if (self && tt == q)
        v = P.s2[ia] + P.t2[ia];
    else
        v = cov_entry(g, P.pt(ia), P.s2[ia], P.beta[ia], P.pt(ib), P.s2[ib], P.beta[ib]);
    out[e] = v;
}

template <typename Ti, typename To>
__global__ void k_convert(const Ti* __restrict__ in, To* __restrict__ out, long n) {
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        out[i] = (To)in[i];
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
void launch_fields(const Geom& g, const FieldParams& fp, const double* c0, const double* c1, const double* c2,
                   long n, double* s2, double* beta, double* t2, cudaStream_t st) {
    if (n <= 0) return;
    k_fields<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, fp, c0, c1, c2, n, s2, beta, t2);
}
template <typename T>
int launch_prior_level(const Geom& g, const DevTree<T>& t, int m, int grid, cudaStream_t st, CovTiming* tm) {
    auto mark = [&](cudaEvent_t e) {
        if (tm->capturing) cudaEventRecordWithFlags(e, st, cudaEventRecordExternal);
        else cudaEventRecord(e, st);
    };
    const long cnt = level_count(t.J, m);
    const long per_region = (long)(m + 1) * t.r * t.r;
    long per = t.cbuf_elems / per_region;  // regions whose blocks fit the buffer at once
    if (per < 1) per = 1;
    int launches = 0;
    for (long loc0 = 0; loc0 < cnt; loc0 += per) {
        const long n = cnt - loc0 < per ? cnt - loc0 : per;
        const long nb = n * (m + 1);
        const long cov_grid = (long)grid * 16;  // 16 per region-kernel slot: 32 CTAs per SM
        const bool timed = tm && tm->used < tm->cap;
        if (tm && !timed) tm->overflow = true;
        if (timed) mark(tm->ev[2 * tm->used]);
        launch_cov_level<T>(g, t, m, loc0, n, (unsigned)(nb < cov_grid ? nb : cov_grid), st);
        if (timed) mark(tm->ev[2 * tm->used++ + 1]);
        k_prior_level<T><<<(unsigned)(n < grid ? n : grid), kThreads, sizeof(LaSmem<T>), st>>>(g, t, m, loc0, n,
                                                                                                t.cbuf);
        launches += 2;
    }
    return launches;
}
template <typename T>
void launch_posterior_level(const Geom& g, const DevTree<T>& t, int m, int grid, bool keep, cudaStream_t st) {
    long cnt = level_count(t.J, m);
    k_posterior_level<T><<<(unsigned)(cnt < grid ? cnt : grid), kThreads, sizeof(LaSmem<T>), st>>>(g, t, m, keep ? 1 : 0);
}
template <typename T>
void launch_predict(const Geom& g, const DevTree<T>& t, int grid, cudaStream_t st) {
    const long cnt2 = level_count(t.J, t.M - 2);
    k_predict<T><<<(unsigned)(cnt2 < grid ? cnt2 : grid), kThreads, sizeof(LaSmem<T>), st>>>(g, t);
}
template <typename T>
void launch_reduce(const DevTree<T>& t, double* out, cudaStream_t st) {
    k_reduce<T><<<1, kThreads, sizeof(LaSmem<T>), st>>>(t, out);
}
template <typename T>
void launch_sample(const DevTree<T>& t, const double* z_int, const double* z_obs, double* y_out, int grid,
                   cudaStream_t st) {
    k_sample<T><<<(unsigned)(t.n_fin < grid ? t.n_fin : grid), kThreads, sizeof(LaSmem<T>), st>>>(t, z_int, z_obs, y_out);
}
void launch_cov_block(const Geom& g, const PointSet& P, long a0, int na, long b0, int nb, bool self, double* out,
                      cudaStream_t st) {
    long n = (long)na * nb;
    if (n <= 0) return;
    k_cov_block<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, P, a0, na, b0, nb, self ? 1 : 0, out);
}

template <typename Ti, typename To>
void launch_convert(const Ti* in, To* out, long n, cudaStream_t st) {
    if (n <= 0) return;
    long blocks = (n + 255) / 256;
    k_convert<Ti, To><<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, st>>>(in, out, n);
}
template void launch_convert<float, double>(const float*, double*, long, cudaStream_t);
template void launch_convert<double, float>(const double*, float*, long, cudaStream_t);

template <typename T>
static cudaError_t prepare_type() {
    const int bytes = (int)sizeof(LaSmem<T>);
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* fn) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
    set((const void*)k_prior_level<T>);
    set((const void*)k_posterior_level<T>);
    set((const void*)k_predict<T>);
    set((const void*)k_reduce<T>);
    set((const void*)k_sample<T>);
    return e;
}

cudaError_t set_gemm_tiles(const int nw[3]) { return cudaMemcpyToSymbol(c_gemm_nw, nw, 3 * sizeof(int)); }

cudaError_t prepare_kernels() {
    cudaError_t e = prepare_type<double>();
    if (e == cudaSuccess) e = prepare_type<float>();
    return e == cudaSuccess ? prepare_finest() : e;
}

#define MRA_INSTANTIATE(T)                                                                                   \
    template int launch_prior_level<T>(const Geom&, const DevTree<T>&, int, int, cudaStream_t, CovTiming*); \
    template void launch_posterior_level<T>(const Geom&, const DevTree<T>&, int, int, bool, cudaStream_t);  \
    template void launch_predict<T>(const Geom&, const DevTree<T>&, int, cudaStream_t);                     \
    template void launch_reduce<T>(const DevTree<T>&, double*, cudaStream_t);                               \
    template void launch_sample<T>(const DevTree<T>&, const double*, const double*, double*, int, cudaStream_t);
MRA_INSTANTIATE(double)
MRA_INSTANTIATE(float)

}  // namespace mra
