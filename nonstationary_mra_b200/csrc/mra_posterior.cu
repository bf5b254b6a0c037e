// Posterior of the MRA hot path (...-posterior-inference.cpp:14-265,
// class_approximation.cpp:186-306), one tree level at a time.
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
//
// A level's dense regions and, where the context keeps at most 128 rows in factored
// form (MRA_FACTORED_MAX; 2r by default, so r <= 64), its factored ones run tile by
// tile, in launches split by what is independent (k_dense_*, k_fact_*).  With a larger
// limit all factored regions, whatever their rows, take one CTA each from a queue
// (k_posterior_factored).  Dense:
//   k_dense_gather   slices (j, k) of the summed children contributions, and
//                    L L^T + A_(m,m): one CTA per tile of a slice
//   k_dense_factor   L~ with its inverse, v, the log-lik term: one CTA per region
//   k_dense_solve    G_j = L~^{-1} A_(j,m)^T
//   k_dense_out      A~_(j,k) = A_(j,k) - G_j^T G_k,  w~_j = w_j - G_j^T v
// One CTA per dense region did all of this in sequence before: a top level of a
// few regions left the chip to as many CTAs (100 to 900 us per level), and a
// clustered region's thousands of rows were summed by one (1.6 of 3.7 ms of the
// posterior of a clustered 65,536-point evaluation in one launch).
#include <algorithm>

#include "mra_kernels.cuh"
#include "mra_tile.cuh"

namespace mra {

// ---------------------------------------------------------------------------
// factored regions of a context that keeps more than 128 rows in factored form
// ---------------------------------------------------------------------------
// The products of the posterior steps go through a separate function: the
// steps keep many values live across their products, and inlined there the
// product loops would share (and spill) their registers.
template <bool TA, bool TB, bool ONE_TILE = false>
__device__ __noinline__ void gemm_call(int M, int N, int K, double alpha, const double* A, long lda, const double* B,
                                       long ldb, double beta, double* C, long ldc, LaSmem<double>& sm) {
    gemm<double, TA, TB, ONE_TILE>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, sm);
}

// Factored input (F: n rows of width (m+1) r, row stride ldF; f: n doubles).
// Writes F' (n rows of width m r) to Fo and f' to fo when m > 0.
__device__ __noinline__ void factored_step(const DevTree<double>& t, int m, long i, int n, const double* F, long ldF,
                                           const double* f, double* Fo, double* fo, bool keep, double* ws, double* wsd,
                                           LaSmem<double>& sm, double& dterm) {
    const int r = t.r;
    const long rr = (long)r * r, mr = (long)m * r;
    const double* Li = t.Lprior + i * rr;
    double* Y = ws;                  // r x n
    double* S = ws + (long)r * n;    // n x n
    double* Rinv = S + (long)n * n;  // n x n (n <= 128)
    // Y = L_i^{-1} F_m^T as a product with the stored inverse of the prior factor
    gemm_call<false, false>(r, n, r, 1.0, t.Pinv + i * rr, r, F + mr, ldF, 0.0, Y, r, sm);
    gemm_call<true, false>(n, n, r, 1.0, Y, r, Y, r, 0.0, S, n, sm);
    for (int q = threadIdx.x; q < n; q += kThreads) S[q + (long)q * n] += 1.0;
    __syncthreads();
    double ld = 0.0;
    const bool small = n <= 128;
    int info = potrf_lower<double>(n, S, n, sm, &ld, small ? Rinv : nullptr, n);
    double* fp = m > 0 ? fo : wsd;
    double part = 0.0;
    for (int q = threadIdx.x; q < n; q += kThreads) {
        fp[q] = f[q];
        part += f[q] * f[q];
    }
    double ff = cta_sum(part, sm);
    if (small) trmv_lower_inv<double>(n, Rinv, n, fp, fp);  // f' = R^{-1} f with the inverse formed above
    else trsv_lower_f64<double>(n, S, n, fp);
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
            gemm_call<false, true>((int)mr, n, n, 1.0, F, ldF, Rinv, n, 0.0, Fo, mr, sm);
        } else {
            for (long e = threadIdx.x; e < mr * n; e += kThreads) {
                long x = e % mr, q = e / mr;
                Fo[q * mr + x] = F[q * ldF + x];
            }
            __syncthreads();
            trsm_right_lower_trans<double>((int)mr, n, S, n, Fo, mr, sm);
        }
    }
    if (keep) {
        // predictive factors of the region: L~ L~^T = L L^T + F_m^T F_m, v = L~^{-1} F_m^T f,
        // G = L~^{-1} F_m^T F_{0..m-1}
        double* Lt = t.Lpost + i * rr;
        gemm_call<false, true>(r, r, r, 1.0, Li, r, Li, r, 0.0, Lt, r, sm);
        gemm_call<false, true>(r, r, n, 1.0, F + mr, ldF, F + mr, ldF, 1.0, Lt, r, sm);
        double* Lti = t.Lpinv ? t.Lpinv + i * rr : nullptr;  // L~^{-1}, kept for prediction
        int info2 = potrf_lower<double>(r, Lt, r, sm, nullptr, Lti, r);
        double* v = t.vpost + i * r;
        for (int tt = threadIdx.x; tt < r; tt += kThreads) {
            double s = 0.0;
            for (int q = 0; q < n; ++q) s += F[(long)q * ldF + mr + tt] * f[q];
            v[tt] = s;
        }
        __syncthreads();
        if (Lti) trmv_lower_inv<double>(r, Lti, r, v, v);
        else trsv_lower_f64<double>(r, Lt, r, v);
        if (m > 0) {
            double* Gi = t.G + t.u_off[m] + (i - t.lstart[m]) * mr * r;
            gemm_call<false, true>(r, (int)mr, n, 1.0, F + mr, ldF, F, ldF, 0.0, Gi, r, sm);
            // G = L~^{-1} G in place: one row tile (r <= 64) reads all of its
            // column block before writing it
            if (Lti) gemm_call<false, false>(r, (int)mr, r, 1.0, Lti, r, Gi, r, 0.0, Gi, r, sm);
            else trsm_left_lower<double>(r, (int)mr, Lt, r, Gi, r, sm);
        }
        if (info2 && threadIdx.x == 0) report_error(t.err, i);
    }
}

// Regions from a shared counter, most expensive first.
__global__ void __launch_bounds__(kThreads, 2) k_posterior_factored(DevTree<double> t, int m, int keep) {
    LaSmem<double>& sm = la_smem<double>();
    const int r = t.r;
    const long mr1 = (long)(m + 1) * r;
    const long s0 = t.lstart[m], nd = t.n_dense[m];
    const long cnt = level_count(t.J, m) - (m == t.M - 2 && !keep ? t.n_fused : 0);
    double* ws = t.ws + blockIdx.x * t.ws_stride;
    double* wsd = t.wsd + blockIdx.x * t.wsd_stride;
    // the children's rows: B^, y~ of the finest level, else F, f of the level below
    const double* Fin = m == t.M - 2 ? t.Bhat : t.Fbuf[(m + 1) & 1];
    const double* fin = m == t.M - 2 ? t.yt : t.fbuf[(m + 1) & 1];
    __shared__ long s_loc;
    for (;;) {
        __syncthreads();  // every thread has read the previous s_loc
        if (threadIdx.x == 0) {
            const long q = nd + atomicAdd(&t.queue[kQueuePost + m], 1);
            s_loc = q < cnt ? t.post_order[s0 + q] : -1;
        }
        __syncthreads();
        const long loc = s_loc;
        if (loc < 0) break;
        const long i = s0 + loc;
        if (skipped(t, i)) continue;
        double dterm = 0.0;
        const long lo = t.sub_lo[i];
        const int n = (int)(t.sub_hi[i] - lo);
        double* Fo = m > 0 ? t.Fbuf[m & 1] + lo * (long)m * r : nullptr;
        double* fo = m > 0 ? t.fbuf[m & 1] + lo : nullptr;
        factored_step(t, m, i, n, Fin + lo * mr1, mr1, fin + lo, Fo, fo, keep != 0, ws, wsd, sm, dterm);
        if (threadIdx.x == 0) t.dpost[i] = dterm;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// dense regions
// ---------------------------------------------------------------------------
// A launch takes regions q0 .. of the level's dense list.  Slices (j, k < m) are
// summed straight into the region's output block (aout) and updated there; the
// slices (j, m), G and the inverse of L~ live in a scratch block per region (the
// prior's covariance buffer, idle by now).
struct DenseArgs {
    int m, keep;
    int col;      // predictive factors of factored regions: only the slices (j, m), from the region's own rows
    long q0;      // first region of the launch in the level's list (post_order)
    double* scr;  // scratch of region q0
    long per;     // doubles of scratch per region: m slices (j, m), m blocks G, the inverse
};

__device__ __forceinline__ double* dense_G(const DevTree<double>& t, const DenseArgs& a, long q, long i) {
    const long rr = (long)t.r * t.r;
    return a.keep ? t.G + t.u_off[a.m] + (i - t.lstart[a.m]) * (long)a.m * rr
                  : a.scr + q * a.per + (long)a.m * rr;
}
__device__ __forceinline__ double* dense_inv(const DevTree<double>& t, const DenseArgs& a, long q, long i) {
    const long rr = (long)t.r * t.r;
    return a.keep && t.Lpinv ? t.Lpinv + i * rr : a.scr + q * a.per + 2L * a.m * rr;
}

template <int TS>
__global__ void __launch_bounds__(Tile<TS>::NT, Tile<TS>::CTAS) k_dense_gather(DevTree<double> t, DenseArgs a, int nt) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using TT = Tile<TS>;
    typename TT::Smem& sm = *reinterpret_cast<typename TT::Smem*>(la_dyn_smem);
    const int r = t.r, m = a.m;
    const long rr = (long)r * r, mr1 = (long)(m + 1) * r;
    const bool vec = r % 2 == 0;
    const int ns = (int)n_slices(m + 1), tasks = a.col ? m + 1 : ns, nt2 = nt * nt;
    const long q = blockIdx.x / (tasks * nt2);
    int s = (int)(blockIdx.x - q * (tasks * nt2));
    const int ti = s % nt2 / nt, tj = s % nt;
    s /= nt2;
    int j = a.col ? s : 0, k = m;  // slice s = (j, k), j <= k <= m, row by row; a.col: (s, m)
    if (!a.col) {
        while (s >= m + 1 - j) s -= m + 1 - j, ++j;
        k = j + s;
    }
    const long i = t.lstart[m] + t.post_order[t.lstart[m] + a.q0 + q];
    if (skipped(t, i)) return;
    const int r0 = ti * TS, c0 = tj * TS;
    const int M = min(TS, r - r0), N = min(TS, r - c0);
    typename TT::Acc acc;
    TT::zero(acc);
    const bool sum_w = j == k && ti == tj;  // this tile also sums w_j
    constexpr int WG = TT::NT / TS;
    const int wx = threadIdx.x % TS, wg = threadIdx.x / TS;
    double w = 0.0;
    auto rows = [&](const double* F, const double* f, int n) {  // n factored rows
        if (n == 0) return;
        TT::template product<false, false>(acc, sm, F + (long)j * r + r0, mr1, M, F + (long)k * r + c0, mr1, N, n, vec,
                                           vec);
        if (sum_w && wx < M) {
#pragma unroll 4
            for (int x = wg; x < n; x += WG) w += F[(long)x * mr1 + j * r + r0 + wx] * f[x];
        }
    };
    if (m == t.M - 2 || a.col) {
        const long lo = t.sub_lo[i];
        rows((m == t.M - 2 ? t.Bhat : t.Fbuf[(m + 1) & 1]) + lo * mr1, (m == t.M - 2 ? t.yt : t.fbuf[(m + 1) & 1]) + lo,
             (int)(t.sub_hi[i] - lo));
    } else {
        const double* Fin = t.Fbuf[(m + 1) & 1];
        const double* fin = t.fbuf[(m + 1) & 1];
        for (int cc = 1; cc <= t.J; ++cc) {
            const long c = i * t.J + cc;
            if (t.factored[c]) {
                // factored children with adjacent rows are summed together
                const long lo = t.sub_lo[c];
                long hi = t.sub_hi[c], cl = c;
                while (cc < t.J && t.factored[cl + 1] && t.sub_lo[cl + 1] == hi) {
                    ++cc;
                    ++cl;
                    hi = t.sub_hi[cl];
                }
                rows(Fin + lo * mr1, fin + lo, (int)(hi - lo));
            } else {
                const long cl = t.dslot[c];
                TT::add(acc, 1.0, t.aout[(m + 1) & 1] + (cl * ns + slice_index(m + 1, j, k)) * rr + r0 + (long)c0 * r, r, M,
                        N);
                if (sum_w && wg == 0 && wx < M) w += t.wout[(m + 1) & 1][cl * mr1 + j * r + r0 + wx];
            }
        }
    }
    double* dst;
    if (k < m) {
        dst = t.aout[m & 1] + (t.dslot[i] * n_slices(m) + slice_index(m, j, k)) * rr;
    } else if (j < m) {
        dst = a.scr + q * a.per + (long)j * rr;
    } else {  // L~ L~^T = L L^T + A_(m,m)
        const double* Li = t.Lprior + i * rr;
        TT::template product<false, false>(acc, sm, Li + r0, r, M, Li + c0, r, N, r, vec, vec);
        dst = t.Lpost + i * rr;
    }
    TT::store(acc, 1.0, dst + r0 + (long)c0 * r, r, M, N);
    if (sum_w) {
        double* part = &sm.A[0][0];
        part[wg * TS + wx] = w;
        __syncthreads();
        if (wg == 0 && wx < M) {
            double sum = 0.0;
            for (int g = 0; g < WG; ++g) sum += part[g * TS + wx];
            double* wd = j < m ? t.wout[m & 1] + t.dslot[i] * (long)m * r + (long)j * r : t.vpost + i * r;
            wd[r0 + wx] = sum;
        }
    }
}

// L~ in place of L L^T + A_(m,m), its inverse (r <= 128), v = L~^{-1} w_m (w_m in vpost).
// MID: 64 < r <= 128, on Potrf128Smem.
template <bool MID>
__global__ void __launch_bounds__(kThreads, MID ? 1 : 2) k_dense_factor(DevTree<double> t, DenseArgs a) {
    LaSmem<double>& sm = la_smem<double>();
    const int r = t.r;
    const long q = blockIdx.x;
    const long i = t.lstart[a.m] + t.post_order[t.lstart[a.m] + a.q0 + q];
    if (skipped(t, i)) return;
    double* Lt = t.Lpost + i * (long)r * r;
    double* X = r <= 128 ? dense_inv(t, a, q, i) : nullptr;
    double ld = 0.0;
    const int info = MID ? potrf_128(r, Lt, r, &ld, X, r) : potrf_lower<double>(r, Lt, r, sm, &ld, X, r);
    double* v = t.vpost + i * r;
    if (X) trmv_lower_inv<double>(r, X, r, v, v);
    else trsv_lower_f64<double>(r, Lt, r, v);
    double part = 0.0;
    for (int e = threadIdx.x; e < r; e += kThreads) part += v[e] * v[e];
    const double vv = cta_sum(part, sm);
    if (threadIdx.x == 0) {
        if (!a.col) t.dpost[i] = ld - t.ldprior[i] - vv;
        if (info) report_error(t.err, i);
    }
}

// G_j = L~^{-1} A_(j,m)^T, one CTA per tile (r <= 128).
template <int TS>
__global__ void __launch_bounds__(Tile<TS>::NT, Tile<TS>::CTAS) k_dense_solve(DevTree<double> t, DenseArgs a, int nt) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using TT = Tile<TS>;
    typename TT::Smem& sm = *reinterpret_cast<typename TT::Smem*>(la_dyn_smem);
    const int r = t.r, m = a.m;
    const long rr = (long)r * r;
    const bool vec = r % 2 == 0;
    const int nt2 = nt * nt;
    const long q = blockIdx.x / (m * nt2);
    const int s = (int)(blockIdx.x - q * (m * nt2));
    const int j = s / nt2, ti = s % nt2 / nt, tj = s % nt;
    const long i = t.lstart[m] + t.post_order[t.lstart[m] + a.q0 + q];
    if (skipped(t, i)) return;
    const int r0 = ti * TS, c0 = tj * TS;
    const int M = min(TS, r - r0), N = min(TS, r - c0);
    typename TT::Acc acc;
    TT::zero(acc);
    // the inverse is lower triangular: rows r0 .. r0 + M - 1 end at column r0 + M - 1
    TT::template product<false, false>(acc, sm, dense_inv(t, a, q, i) + r0, r, M, a.scr + q * a.per + (long)j * rr + c0,
                                       r, N, r0 + M, vec, vec);
    TT::store(acc, 1.0, dense_G(t, a, q, i) + (long)j * rr + r0 + (long)c0 * r, r, M, N);
}

// The same for r > 128: triangular solves, one CTA per region.
__global__ void __launch_bounds__(kThreads, 2) k_dense_solve_any(DevTree<double> t, DenseArgs a) {
    LaSmem<double>& sm = la_smem<double>();
    const int r = t.r, m = a.m;
    const long rr = (long)r * r, mr = (long)m * r;
    const long q = blockIdx.x;
    const long i = t.lstart[m] + t.post_order[t.lstart[m] + a.q0 + q];
    if (skipped(t, i)) return;
    const double* A = a.scr + q * a.per;
    double* G = dense_G(t, a, q, i);
    for (long e = threadIdx.x; e < mr * r; e += kThreads) {
        const long j = e / rr, w = e % rr;
        G[e] = A[j * rr + w / r + (w % r) * r];
    }
    __syncthreads();
    trsm_left_lower<double>(r, (int)mr, t.Lpost + i * rr, r, G, r, sm);
}

template <int TS>
__global__ void __launch_bounds__(Tile<TS>::NT, Tile<TS>::CTAS) k_dense_out(DevTree<double> t, DenseArgs a, int nt) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using TT = Tile<TS>;
    typename TT::Smem& sm = *reinterpret_cast<typename TT::Smem*>(la_dyn_smem);
    const int r = t.r, m = a.m;
    const long rr = (long)r * r;
    const bool vec = r % 2 == 0;
    const int ns = (int)n_slices(m), nt2 = nt * nt;
    const long q = blockIdx.x / (ns * nt2);
    int s = (int)(blockIdx.x - q * (ns * nt2));
    const int ti = s % nt2 / nt, tj = s % nt;
    s /= nt2;
    int j = 0;
    while (s >= m - j) s -= m - j, ++j;
    const int k = j + s;
    const long i = t.lstart[m] + t.post_order[t.lstart[m] + a.q0 + q];
    if (skipped(t, i)) return;
    const int r0 = ti * TS, c0 = tj * TS;
    const int M = min(TS, r - r0), N = min(TS, r - c0);
    const double* G = dense_G(t, a, q, i);
    double* A = t.aout[m & 1] + (t.dslot[i] * n_slices(m) + slice_index(m, j, k)) * rr + r0 + (long)c0 * r;
    typename TT::Acc acc;
    TT::zero(acc);
    TT::add(acc, -1.0, A, r, M, N);
    TT::template product<true, true>(acc, sm, G + (long)j * rr + (long)r0 * r, r, M, G + (long)k * rr + (long)c0 * r, r, N,
                                     r, vec, vec);
    TT::store(acc, -1.0, A, r, M, N);
    if (j == k && ti == tj) {
        constexpr int WG = TT::NT / TS;
        const int wx = threadIdx.x % TS, wg = threadIdx.x / TS;
        const double* v = t.vpost + i * r;
        double w = 0.0;
        if (wx < M) {
#pragma unroll 4
            for (int x = wg; x < r; x += WG) w += G[(long)j * rr + x + (long)(r0 + wx) * r] * v[x];
        }
        double* part = &sm.A[0][0];
        part[wg * TS + wx] = w;
        __syncthreads();
        if (wg == 0 && wx < M) {
            double sum = 0.0;
            for (int g = 0; g < WG; ++g) sum += part[g * TS + wx];
            t.wout[m & 1][t.dslot[i] * (long)m * r + (long)j * r + r0 + wx] -= sum;
        }
    }
}

// ---------------------------------------------------------------------------
// factored regions of a context that keeps at most 128 rows in factored form, in tiles
// ---------------------------------------------------------------------------
// k_fact_y       Y = L^{-1} F_m^T                      one CTA per tile
// k_fact_factor  R R^T = I + Y^T Y with R^{-1}, f'     one CTA per region
// k_fact_out     F' = F_{0..m-1} R^{-T}                one CTA per tile
// In one CTA per region these were a chain of small products between barriers
// (tensor pipe 22% busy); the two wide ones now fill the chip.  4,096 regions of
// about 64 rows and 64 knots with 6 ancestors: 2.09 -> 1.5 ms.
struct FactArgs {
    int m, keep;
    long q0;      // first region of the launch in the level's list (post_order)
    double* scr;  // scratch of region q0: Y [r x n], S [n x n], R^{-1} [n x n]
    long per;
};

template <int TS>
__global__ void __launch_bounds__(Tile<TS>::NT, Tile<TS>::CTAS) k_fact_y(DevTree<double> t, FactArgs a, int nt, int nc) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using TT = Tile<TS>;
    typename TT::Smem& sm = *reinterpret_cast<typename TT::Smem*>(la_dyn_smem);
    const int r = t.r, m = a.m;
    const long mr1 = (long)(m + 1) * r;
    const long q = blockIdx.x / (nt * nc);
    const int s = (int)(blockIdx.x - q * (nt * nc)), r0 = s / nc * TS, c0 = s % nc * TS;
    const long i = t.lstart[m] + t.post_order[t.lstart[m] + a.q0 + q];
    const long lo = t.sub_lo[i];
    const int n = (int)(t.sub_hi[i] - lo);
    if (c0 >= n || skipped(t, i)) return;
    const int M = min(TS, r - r0), N = min(TS, n - c0);
    const double* F = (m == t.M - 2 ? t.Bhat : t.Fbuf[(m + 1) & 1]) + lo * mr1;
    const bool vec = r % 2 == 0;
    typename TT::Acc acc;
    TT::zero(acc);
    // the factor's inverse is lower triangular: rows up to r0 + M - 1
    TT::template product<false, true>(acc, sm, t.Pinv + i * (long)r * r + r0, r, M, F + (long)c0 * mr1 + (long)m * r, mr1, N,
                                      r0 + M, vec && M % 2 == 0, vec && (r0 + M) % 2 == 0);
    TT::store(acc, 1.0, a.scr + q * a.per + r0 + (long)c0 * r, r, M, N);
}

// MID: regions of 65 to 128 rows, on Potrf128Smem (the level's list starts with the
// largest); otherwise the others.
template <bool MID>
__global__ void __launch_bounds__(kThreads, MID ? 1 : 2) k_fact_factor(DevTree<double> t, FactArgs a) {
    LaSmem<double>& sm = la_smem<double>();
    const int r = t.r, m = a.m;
    const long q = blockIdx.x;
    const long i = t.lstart[m] + t.post_order[t.lstart[m] + a.q0 + q];
    if (skipped(t, i)) return;
    const long lo = t.sub_lo[i];
    const int n = (int)(t.sub_hi[i] - lo);
    if (MID != (n > 64)) return;
    if (n == 0) {
        if (threadIdx.x == 0) t.dpost[i] = 0.0;
        return;
    }
    double* Y = a.scr + q * a.per;
    double* S = Y + (long)r * n;
    double* X = S + (long)n * n;
    gemm<double, true, false>(n, n, r, 1.0, Y, r, Y, r, 0.0, S, n, sm);
    for (int e = threadIdx.x; e < n; e += kThreads) S[e + (long)e * n] += 1.0;
    __syncthreads();
    double ld = 0.0;
    const int info = MID ? potrf_128(n, S, n, &ld, X, n) : potrf_small(n, S, n, sm, &ld, X, n);
    // f' = R^{-1} f
    const double* f = (m == t.M - 2 ? t.yt : t.fbuf[(m + 1) & 1]) + lo;
    double* fp = m > 0 ? t.fbuf[m & 1] + lo : t.wsd;  // level 0 has one region
    trmv_lower_inv<double>(n, X, n, fp, f);
    double part = 0.0;
    for (int e = threadIdx.x; e < n; e += kThreads) part += f[e] * f[e] - fp[e] * fp[e];
    const double dd = cta_sum(part, sm);
    if (threadIdx.x == 0) {
        t.dpost[i] = ld - dd;
        if (info) report_error(t.err, i);
    }
}

template <int TS>
__global__ void __launch_bounds__(Tile<TS>::NT, Tile<TS>::CTAS) k_fact_out(DevTree<double> t, FactArgs a, int nx, int nc) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using TT = Tile<TS>;
    typename TT::Smem& sm = *reinterpret_cast<typename TT::Smem*>(la_dyn_smem);
    const int r = t.r, m = a.m;
    const long mr = (long)m * r, mr1 = mr + r;
    const long q = blockIdx.x / (nx * nc);
    const int s = (int)(blockIdx.x - q * (nx * nc)), x0 = s / nc * TS, c0 = s % nc * TS;
    const long i = t.lstart[m] + t.post_order[t.lstart[m] + a.q0 + q];
    const long lo = t.sub_lo[i];
    const int n = (int)(t.sub_hi[i] - lo);
    if (c0 >= n || skipped(t, i)) return;
    const int M = (int)min((long)TS, mr - x0), N = min(TS, n - c0);
    const double* F = (m == t.M - 2 ? t.Bhat : t.Fbuf[(m + 1) & 1]) + lo * mr1;
    const double* X = a.scr + q * a.per + (long)r * n + (long)n * n;
    const bool vec = r % 2 == 0;
    typename TT::Acc acc;
    TT::zero(acc);
    // R^{-1} is lower triangular: its rows c0 .. c0 + N - 1 end at column c0 + N - 1
    TT::template product<false, false>(acc, sm, F + x0, mr1, M, X + c0, n, N, c0 + N, vec && M % 2 == 0,
                                       n % 2 == 0 && vec);
    TT::store(acc, 1.0, t.Fbuf[m & 1] + lo * mr + x0 + (long)c0 * mr, mr, M, N);
}

// ---------------------------------------------------------------------------
// launcher
// ---------------------------------------------------------------------------
static void launch_dense_factor(const DevTree<double>& t, const DenseArgs& a, long n, cudaStream_t st) {
    if (t.r > 64 && t.r <= 128) k_dense_factor<true><<<(unsigned)n, kThreads, sizeof(Potrf128Smem), st>>>(t, a);
    else k_dense_factor<false><<<(unsigned)n, kThreads, sizeof(LaSmem<double>), st>>>(t, a);
}

template <int TS>
static int launch_dense(const DevTree<double>& t, int m, long elems, bool keep, cudaStream_t st) {
    const int nt = (t.r + TS - 1) / TS, nt2 = nt * nt;
    const size_t sb = sizeof(typename Tile<TS>::Smem);
    DenseArgs a{m, keep ? 1 : 0, 0, 0, t.cbuf, dense_scratch(m, t.r)};
    const long most = elems / a.per;  // regions whose scratch fits at once
    int launches = 0;
    for (a.q0 = 0; a.q0 < t.n_dense[m]; a.q0 += most) {
        const long n = t.n_dense[m] - a.q0 < most ? t.n_dense[m] - a.q0 : most;
        k_dense_gather<TS><<<(unsigned)(n * n_slices(m + 1) * nt2), Tile<TS>::NT, sb, st>>>(t, a, nt);
        launch_dense_factor(t, a, n, st);
        launches += 2;
        if (m == 0) continue;
        if (t.r <= 128) k_dense_solve<TS><<<(unsigned)(n * m * nt2), Tile<TS>::NT, sb, st>>>(t, a, nt);
        else k_dense_solve_any<<<(unsigned)n, kThreads, sizeof(LaSmem<double>), st>>>(t, a);
        k_dense_out<TS><<<(unsigned)(n * n_slices(m) * nt2), Tile<TS>::NT, sb, st>>>(t, a, nt);
        launches += 2;
    }
    return launches;
}

template <int TS>
static int launch_factored(const DevTree<double>& t, int m, long nf, double* scr, long elems, bool keep, cudaStream_t st) {
    const size_t sb = sizeof(typename Tile<TS>::Smem);
    const int nt = (t.r + TS - 1) / TS, nc = (t.tf + TS - 1) / TS, nx = (int)(((long)m * t.r + TS - 1) / TS);
    const long per = fact_scratch(m, t.r, t.tf, keep);
    const long most = elems / per;
    int launches = 0;
    for (long k0 = 0; k0 < nf; k0 += most) {
        const long n = nf - k0 < most ? nf - k0 : most;
        const FactArgs a{m, keep ? 1 : 0, t.n_dense[m] + k0, scr, per};
        // (MRA_FACTORED_MAX = 0 leaves only regions without rows)
        if (nc > 0) k_fact_y<TS><<<(unsigned)(n * nt * nc), Tile<TS>::NT, sb, st>>>(t, a, nt, nc);
        // the list is by cost, and so by rows: the first n_mid regions hold more than 64
        const long mid = t.n_mid[m] - k0 < n ? t.n_mid[m] - k0 : n;
        if (mid > 0) {
            k_fact_factor<true><<<(unsigned)mid, kThreads, sizeof(Potrf128Smem), st>>>(t, a);
            ++launches;
        }
        k_fact_factor<false><<<(unsigned)n, kThreads, sizeof(LaSmem<double>), st>>>(t, a);
        launches += 2;
        if (m > 0 && nc > 0) {
            k_fact_out<TS><<<(unsigned)(n * nx * nc), Tile<TS>::NT, sb, st>>>(t, a, nx, nc);
            ++launches;
        }
        if (!keep) continue;
        // predictive factors: L~ L~^T = L L^T + F_m^T F_m, v = L~^{-1} F_m^T f, G = L~^{-1} F_m^T F_{0..m-1}
        const DenseArgs d{m, 1, 1, a.q0, scr, per};
        k_dense_gather<TS><<<(unsigned)(n * (m + 1) * nt * nt), Tile<TS>::NT, sb, st>>>(t, d, nt);
        launch_dense_factor(t, d, n, st);
        launches += 2;
        if (m == 0) continue;
        if (t.r <= 128) k_dense_solve<TS><<<(unsigned)(n * m * nt * nt), Tile<TS>::NT, sb, st>>>(t, d, nt);
        else k_dense_solve_any<<<(unsigned)n, kThreads, sizeof(LaSmem<double>), st>>>(t, d);
        ++launches;
    }
    return launches;
}

template <int TS>
static int launch_level(const DevTree<double>& t, int m, long nf, int grid, bool keep, cudaStream_t st, const Fork& fk) {
    int launches = 0;
    // factored regions beside the dense ones (both need only the level below)
    const bool both = nf > 0 && t.n_dense[m] > 0;
    const bool tiles = t.tf <= 128;
    cudaStream_t sf = both ? fk.side : st;
    const long need_d = dense_scratch(m, t.r), need_f = fact_scratch(m, t.r, t.tf, keep);
    long elems_f = tiles ? t.cbuf_elems : 0, elems_d = t.cbuf_elems;
    if (both && tiles) {
        // the scratch in two: half each, or what one factored region needs, but never less for the dense ones than
        // one of them needs (the buffer holds one of each at least)
        elems_f = std::max(need_f, std::min(t.cbuf_elems / 2, nf * need_f));
        elems_f = std::min(elems_f, t.cbuf_elems - need_d) & ~1L;
        elems_d = (t.cbuf_elems - elems_f) & ~1L;
    }
    // every loop below takes at least one region per turn
    if ((t.n_dense[m] > 0 && elems_d < need_d) || (nf > 0 && tiles && elems_f < need_f)) return -1;
    if (both) {
        cudaEventRecord(fk.fork, st);
        cudaStreamWaitEvent(fk.side, fk.fork, 0);
    }
    if (t.n_dense[m] > 0) launches += launch_dense<TS>(t, m, elems_d, keep, st);
    if (nf > 0) {
        if (tiles) {
            launches += launch_factored<TS>(t, m, nf, t.cbuf + (both ? elems_d : 0), elems_f, keep, sf);
        } else {
            k_posterior_factored<<<(unsigned)(nf < grid ? nf : grid), kThreads, sizeof(LaSmem<double>), sf>>>(
                t, m, keep ? 1 : 0);
            ++launches;
        }
    }
    if (both) {
        cudaEventRecord(fk.join, sf);
        cudaStreamWaitEvent(st, fk.join, 0);
    }
    return launches;
}

int launch_posterior_level(const DevTree<double>& t, int m, int grid, bool keep, cudaStream_t st, const Fork& fk) {
    const long nf = level_count(t.J, m) - t.n_dense[m] - (m == t.M - 2 && !keep ? t.n_fused : 0);
    if (t.r <= 16) return launch_level<16>(t, m, nf, grid, keep, st, fk);
    if (t.r <= 32) return launch_level<32>(t, m, nf, grid, keep, st, fk);
    return launch_level<64>(t, m, nf, grid, keep, st, fk);
}

template <int TS>
static cudaError_t prepare_dense() {
    const int bytes = (int)sizeof(typename Tile<TS>::Smem);
    cudaError_t e = cudaSuccess;
    for (const void* fn : {(const void*)k_dense_gather<TS>, (const void*)k_dense_solve<TS>, (const void*)k_dense_out<TS>,
                           (const void*)k_fact_y<TS>, (const void*)k_fact_out<TS>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e;
}

cudaError_t prepare_posterior() {
    cudaError_t e = prepare_dense<16>();
    if (e == cudaSuccess) e = prepare_dense<32>();
    if (e == cudaSuccess) e = prepare_dense<64>();
    for (const void* fn : {(const void*)k_posterior_factored, (const void*)k_dense_factor<false>,
                           (const void*)k_dense_solve_any, (const void*)k_fact_factor<false>})
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LaSmem<double>));
    for (const void* fn : {(const void*)k_dense_factor<true>, (const void*)k_fact_factor<true>})
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Potrf128Smem));
    return e;
}

cudaError_t set_gemm_tiles_posterior(const int nw[3]) { return cudaMemcpyToSymbol(c_gemm_nw, nw, 3 * sizeof(int)); }

}  // namespace mra
