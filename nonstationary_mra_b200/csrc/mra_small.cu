// Finest regions of few observations (FP64): sibling groups of at most 64
// observations whose regions hold at most 32 each, and single regions of at most
// 64, one CTA per item in tile classes of 16, 32 and 64 observations.
//
// With G = U_S^T U_S (over all ancestors) and G_p its part of the level M-2
// parent p, an item's work needs its rows of U and V once each:
//   Sigma_c = C_c - G_cc per region c,  L_c = chol(Sigma_c),  y~ = L^{-1} y
//   (L block diagonal over the group's regions),  B^ = V L^{-T}.
// For a whole group the level M-2 posterior follows without B^: the parent's rows
// are F_p = B^_p, and L_p^{-1} F_p^T = L_p^{-1} V_p L^{-T} = U_p L^{-T}, so
//   R R^T = I + L^{-1} G_p L^{-T},  f' = R^{-1} y~,
//   F' = R^{-1} F_{0..M-3} = (R^{-1} L^{-1}) V_{0..M-3},
// with one small matrix W = R^{-1} L^{-1} applied to V: no product with the
// parent's factor, and B^ is neither written nor read back.  Prediction, which
// reads B^, and regions whose parent is dense take W = L^{-1} over all rows.
// What bounds it is the stream of U and V (8 KB per observation at 64 knots and 8
// ancestors, F' as much again) behind short serial chains, hence small CTAs, four
// per SM in the classes of 16 and 32.  262,144 observations in 16,384 groups at 64
// knots: 1.3 ms, against 2.9 + 2.3 ms for a group's children with B^ and then the
// parent's posterior from B^ through the general 64-row products.
#include "mra_cond.cuh"

namespace mra {

template <int RC>
struct SmallSmem {
    static constexpr int NT = RC == 64 ? 256 : 128;                  // threads
    static constexpr int CTAS = RC == 64 ? 2 : 4;              // per SM
    static constexpr int LD = RC + 4;
    static constexpr int KD = RC == 64 ? 32 : 64;                    // slab depth of the Gram product
    static constexpr int Z = 2 * RC * KD > RC * LD ? 2 * RC * KD : RC * LD;
    double S[RC * LD];  // Sigma, then H = L^{-1} G_p, then R^{-1}
    double T[RC * LD];  // G_p, then R, then W
    double Z_[Z];       // the two slabs of U, then L^{-1}
    double f[RC];
    double red[NT / 32];
    int flag;
};

// C = A op(B) on n8 x n8 tiles of 8 in shared memory (column-major, row stride LD):
// A lower triangular; BT: op(B) = B^T with B lower triangular and only C's lower
// tiles formed, + I on the diagonal; else op(B) = B (kLowB: lower triangular, C too).
template <int LD, int NT, bool BT, bool kLowB>
__device__ __forceinline__ void small_product(int n8, double* C, const double* A, const double* B) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    for (int e = w; e < n8 * n8; e += NT / 32) {
        const int i = e / n8, j = e - i * n8;
        if ((BT || kLowB) && j > i) continue;
        double acc[2] = {0.0, 0.0};
        const int k_lo = kLowB ? 8 * j : 0, k_hi = 8 * ((BT ? j : i) + 1);
        for (int k = k_lo; k < k_hi; k += 4)
            mma_f64(acc, A[8 * i + g + (k + t) * LD], BT ? B[8 * j + g + (k + t) * LD] : B[k + t + (8 * j + g) * LD]);
#pragma unroll
        for (int h = 0; h < 2; ++h)
            C[8 * i + g + (8 * j + 2 * t + h) * LD] = acc[h] + (BT && i == j && g == 2 * t + h ? 1.0 : 0.0);
    }
}

// C(S_c, S_c) of the small regions, into Lsig: wpr warps per region (8 where regions
// are few: 256 regions of 40 to 64 observations took 60 us with one).
template <int KIND>
__global__ void __launch_bounds__(256) k_cov_group(Geom g, DevTree<double> t, int wpr) {
    const int lane = threadIdx.x & 31;
    const long gw = (long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const long nw = (long)gridDim.x * (blockDim.x / 32) / wpr;
    const int part = (int)(gw % wpr);
    using F = CovForm<KIND>;
    const PointSet& P = t.pts;
    for (long c = gw / wpr; c < t.n_fin; c += nw) {
        const long o0 = t.obs_off[c];
        const int n = (int)(t.obs_off[c + 1] - o0);
        if (n == 0 || n > kFinTile || skipped(t, (long)t.fin_anc[c * t.L + t.L - 1])) continue;
        double* S = t.Lsig + t.lsig_off[c];
        for (int e = 32 * part + lane; e < n * n; e += 32 * wpr) {
            const int i = e % n, j = e / n;
            const long ia = t.obs0 + o0 + i, ib = t.obs0 + o0 + j;
            const double sa = P.s2[ia], ba = P.beta[ia], bb = P.beta[ib];
            double v;
            if (i == j) {
                v = sa + P.t2[ia];
            } else if constexpr (KIND == 0) {
                v = cov_entry(g, P.pt(ia), sa, ba, P.pt(ib), P.s2[ib], bb);
            } else {
                const double ra = F::PREF ? P.ss[ia] : sa, rb = F::PREF ? P.ss[ib] : P.s2[ib];
                auto entry = [&](auto safe) {
                    bool bad = false;
                    v = cov_fast_entry<F::NU, F::PREF, decltype(safe)::value>(
                        P.c0[ia], P.c1[ia], P.c2[ia], 0.5 * (ba * ba), ra * ba, ra, ba, P.c0[ib],
                        P.c1[ib], P.c2[ib], 0.5 * (bb * bb), rb * bb, rb, bb, fabs(g.dist_scale), bad);
                    return bad;
                };
                if (entry(std::false_type())) entry(std::true_type());
            }
            S[e] = v;
        }
    }
}

// Items of one tile class: a value v < J^(M-2) is that sibling group, else the
// finest region v - J^(M-2).
template <int RC, bool EVEN>
__global__ void __launch_bounds__(SmallSmem<RC>::NT, SmallSmem<RC>::CTAS)
    k_finest_small(DevTree<double> t, const int64_t* __restrict__ items, int keep) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using SM = SmallSmem<RC>;
    SM& sm = *reinterpret_cast<SM*>(la_dyn_smem);
    constexpr int NT = SM::NT, LD = SM::LD, KD = SM::KD, NW = NT / 32;
    constexpr int RG = RC / 16, KS = NW / RG, NFC = RC / 8;  // row groups; warps that share a row group's K; column fragments
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, tt = lane & 3;
    const int r = t.r, L = t.L, m = t.M - 2;
    const long Lr = (long)L * r, mr = (long)m * r;
    const long s2 = t.lstart[m], cnt2 = level_count(t.J, m);
    const long item = items[blockIdx.x];
    const bool group = item < cnt2;
    const long clo = group ? t.child_lo[item] : item - cnt2, chi = group ? t.child_hi[item] : clo + 1;
    const long p = group ? s2 + item : (long)t.fin_anc[clo * L + L - 1];
    if (skipped(t, p)) return;
    const long lo = t.obs_off[clo];
    const int np = (int)(t.obs_off[chi] - lo);
    const bool fused = group && !keep && t.factored[p];
    const double* U = t.Ufin + lo * Lr;
    double* V = t.Bhat + lo * Lr;
    double* S = sm.S;
    double* T = sm.T;
    double* Bi = sm.Z_;
    const int n16 = (np + 15) & ~15, n8 = (np + 7) >> 3;

    // G over K in [0, mr) and [mr, Lr): S = -G, T = G_p (lower tiles; T mirrored)
    const int rg = w % RG, ks = w / RG;
    const int sw = cond_swz(g);
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        const long kb = pass ? mr : 0;
        const int K = (int)((pass ? Lr : mr) - kb);
        double acc[2][NFC][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int f = 0; f < NFC; ++f) acc[i][f][0] = acc[i][f][1] = 0.0;
        const int ns = (K + KD - 1) / KD;
        auto issue = [&](int v) {
            if (v < ns) {
                constexpr int PK = EVEN ? KD / 2 : KD, NR = NT / PK;
                const int c = tid % PK, k = v * KD + (EVEN ? 2 * c : c);
                double* sb = sm.Z_ + (v & 1) * (RC * KD);
                for (int i = tid / PK; i < n16; i += NR) {
                    const bool ok = i < np && k < K;
                    const double* src = ok ? U + kb + k + (long)i * Lr : U;
                    double* dst = sb + i * KD + (EVEN ? (c ^ cond_swz(i)) * 2 : ((c >> 1) ^ cond_swz(i)) * 2 + (c & 1));
                    if (EVEN) cp_async16z(dst, src, ok);
                    else cp_async8(dst, src, ok);
                }
            }
            cp_async_commit();
        };
        issue(0);
        for (int v = 0; v < ns; ++v) {
            cp_async_wait<0>();
            __syncthreads();
            issue(v + 1);
            if (16 * rg < np) {
                const double* sb = sm.Z_ + (v & 1) * (RC * KD) + g * KD;
#pragma unroll
                for (int q = ks; q < KD / 8; q += KS) {
                    const int off = ((4 * q + tt) ^ sw) * 2;
                    const double2 x0 = lds2(sb + 16 * rg * KD + off), x1 = lds2(sb + (16 * rg + 8) * KD + off);
#pragma unroll
                    for (int f = 0; f < NFC; ++f) {
                        if (f > 2 * rg + 1) continue;  // lower tiles
                        const double2 y = f == 2 * rg ? x0 : (f == 2 * rg + 1 ? x1 : lds2(sb + 8 * f * KD + off));
                        if (f <= 2 * rg) mma_f64(acc[0][f], x0.x, y.x);
                        mma_f64(acc[1][f], x1.x, y.x);
                        if (f <= 2 * rg) mma_f64(acc[0][f], x0.y, y.y);
                        mma_f64(acc[1][f], x1.y, y.y);
                    }
                }
            }
        }
        for (int q = 0; q < KS; ++q) {  // the K shares of a row group in turn
            __syncthreads();
            if (ks != q || 16 * rg >= np) continue;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int f = 0; f < NFC; ++f) {
                    if (f > 2 * rg + i) continue;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int a = 16 * rg + 8 * i + g, b = 8 * f + 2 * tt + h;
                        double* s = S + a + b * LD;
                        *s = (q > 0 || pass ? *s : 0.0) - acc[i][f][h];
                        if (pass) {
                            double* tp = T + a + b * LD;
                            const double v = (q > 0 ? *tp : 0.0) + acc[i][f][h];
                            *tp = v;
                            if (q == KS - 1 && f < 2 * rg + i) T[b + a * LD] = v;  // diagonal tiles hold both halves
                        }
                    }
                }
        }
    }
    __syncthreads();

    // Sigma_c, L_c, y~ and L^{-1} (into Bi)
    double part = 0.0;  // log-lik terms
    if (group) {
        for (int c = w; c < n16; c += NW)
            for (int i = lane; i < n16; i += 32) Bi[i + c * LD] = 0.0;
        __syncthreads();
        for (long c = clo + w; c < chi; c += NW) {
            const long o0 = t.obs_off[c];
            const int n = (int)(t.obs_off[c + 1] - o0), q0 = (int)(o0 - lo);
            if (n == 0) continue;
            double* Sc = S + q0 * (LD + 1);
            double* Lc = t.Lsig + t.lsig_off[c];
            for (int e = lane; e < n * n; e += 32) {
                const int i = e % n, j = e / n;
                if (i >= j) Sc[i + j * LD] += Lc[e];
            }
            __syncwarp();
            int bad = 0;
            double rk = 0.0;  // 1 / L_kk in lane k
            for (int k = 0; k < n; ++k) {  // lane i owns row i
                const double d = Sc[k + k * LD];
                __syncwarp();
                if (!(d > 0.0)) bad = 1;
                const double rd = rsqrt(d);
                double lik = 0.0;
                if (lane == k) {
                    rk = rd;
                    Sc[k + k * LD] = d * rd;
                } else if (lane > k && lane < n) {
                    lik = Sc[lane + k * LD] * rd;
                    Sc[lane + k * LD] = lik;
                }
                __syncwarp();
                for (int j = k + 1; j < n; ++j)  // uniform trip count across the warp
                    if (lane >= j && lane < n) Sc[lane + j * LD] -= lik * Sc[j + k * LD];
                __syncwarp();
            }
            for (int e = lane; e < n * n; e += 32) {
                const int i = e % n, j = e / n;
                Lc[e] = i >= j ? Sc[i + j * LD] : 0.0;
            }
            double ldp = lane < n ? log(Sc[lane + lane * LD]) : 0.0;
            for (int o = 16; o > 0; o >>= 1) ldp += __shfl_xor_sync(0xffffffffu, ldp, o);
            // column j of L_c^{-1} by lane j; lanes walk the same rows and terms (zeros above the diagonal)
            double* Xc = Bi + q0 * (LD + 1) + (lane < n ? lane : 0) * LD;
            for (int i = 0; i < n; ++i) {
                const double ri = __shfl_sync(0xffffffffu, rk, i);
                double v = 0.0;
                for (int k = 0; k < i; ++k) v += Sc[i + k * LD] * Xc[k];
                if (lane < n) Xc[i] = i == lane ? ri : (i > lane ? -v * ri : 0.0);
            }
            __syncwarp();
            // y~ = L_c^{-1} y: lane i holds row i
            double xl = 0.0;
            const double yl = lane < n ? t.y[o0 + lane] : 0.0;
            for (int k = 0; k < n; ++k) {
                const double yk = __shfl_sync(0xffffffffu, yl, k);
                if (lane < n) xl += Bi[(q0 + lane) + (q0 + k) * LD] * yk;
            }
            if (lane < n) {
                t.yt[o0 + lane] = xl;
                sm.f[q0 + lane] = xl;
            }
            double yy = lane < n ? xl * xl : 0.0;
            for (int o = 16; o > 0; o >>= 1) yy += __shfl_xor_sync(0xffffffffu, yy, o);
            if (lane == 0) part += yy + 2.0 * ldp;
            if (bad && lane == 0) report_error(t.err, t.n_int + c);
        }
    } else {
        double* Lc = t.Lsig + t.lsig_off[clo];
        for (int c = w; c < n16; c += NW)
            for (int i = lane; i < n16; i += 32) {
                if (i < np && c <= i) S[i + c * LD] += Lc[i + (long)c * np];
                if (i >= np) S[i + c * LD] = i == c ? 1.0 : 0.0;
            }
        __syncthreads();
        potrf_core<true, SM, NT, LD>(np, S, Bi, sm);
        for (int c = w; c < np; c += NW)
            for (int i = lane; i < np; i += 32) Lc[i + (long)c * np] = i >= c ? S[i + c * LD] : 0.0;
        if (tid < 64) {
            double s = 0.0;
            if (tid < np) {
                for (int k = 0; k <= tid; ++k) s += Bi[tid + k * LD] * t.y[lo + k];
                t.yt[lo + tid] = s;
                s = s * s + 2.0 * log(S[tid + tid * LD]);
            }
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) part = s;
        }
        if (tid == 0 && sm.flag) report_error(t.err, t.n_int + clo);
        // rows and columns of L^{-1} beyond np (the identity's) do not enter the product below
    }
    __syncthreads();
    if (lane == 0) sm.red[w] = part;
    __syncthreads();
    if (tid == 0) {
        double s = 0.0;
        for (int q = 0; q < NW; ++q) s += sm.red[q];
        t.dchild[clo] = s;
    }

    // the level M-2 posterior of a group
    const double* W = Bi;
    long rows = Lr, ldo = Lr;
    double* out = V;
    if (fused) {
        small_product<LD, NT, false, false>(n8, S, Bi, T);
        __syncthreads();
        small_product<LD, NT, true, false>(n8, T, S, Bi);
        __syncthreads();
        potrf_core<true, SM, NT, LD>(np, T, S, sm);
        double term = 0.0;
        if (tid < np) {
            double fq = 0.0;
            for (int k = 0; k <= tid; ++k) fq += S[tid + k * LD] * sm.f[k];  // f' = R^{-1} y~
            if (m > 0) t.fbuf[m & 1][lo + tid] = fq;
            term = 2.0 * log(T[tid + tid * LD]) - (sm.f[tid] * sm.f[tid] - fq * fq);
        }
        for (int o = 16; o > 0; o >>= 1) term += __shfl_xor_sync(0xffffffffu, term, o);
        __syncthreads();  // R has been read
        if (lane == 0) sm.red[w] = term;
        const int bad = sm.flag;
        small_product<LD, NT, false, true>(n8, T, S, Bi);
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int q = 0; q < NW; ++q) s += sm.red[q];
            t.dpost[p] = s;
            if (bad) report_error(t.err, p);
        }
        W = T;
        rows = mr;
        ldo = mr;
        out = m > 0 ? t.Fbuf[m & 1] + lo * mr : nullptr;
    }

    // out(x, n) = sum_{k <= n} V(x, k) W(n, k): a warp takes 16 rows x at a time straight from
    // memory, rows in pairs (fragment i: row 2g + i); in place for B^
    const int nk = (np + 3) >> 2;
    for (long b = w; b * 16 < rows; b += NW) {
        const long x = b * 16 + 2 * g;
        double acc[2][NFC][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int f = 0; f < NFC; ++f) acc[i][f][0] = acc[i][f][1] = 0.0;
        constexpr int KB = RC == 16 ? 4 : 8;  // loads in flight
#pragma unroll
        for (int k0 = 0; k0 < RC / 4; k0 += KB) {
            if (k0 >= nk) break;
            double2 a[KB];
#pragma unroll
            for (int q = 0; q < KB; ++q) {
                const int k = 4 * (k0 + q) + tt;
                const double* src = V + x + (long)k * Lr;
                a[q] = make_double2(0.0, 0.0);
                if (k < np && x < rows) {
                    if (EVEN) {
                        a[q] = *reinterpret_cast<const double2*>(src);
                    } else {
                        a[q].x = src[0];
                        if (x + 1 < rows) a[q].y = src[1];
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < KB; ++q) {
                if (k0 + q >= nk) break;
                const int k = 4 * (k0 + q);
#pragma unroll
                for (int f = 0; f < NFC; ++f) {
                    if (f < (k0 + q) / 2 || f >= n8) continue;  // W lower triangular
                    const double y = W[8 * f + g + (k + tt) * LD];
                    mma_f64(acc[0][f], a[q].x, y);
                    mma_f64(acc[1][f], a[q].y, y);
                }
            }
        }
        if (!EVEN) __syncwarp();  // in place: every lane has read the rows' pairs
#pragma unroll
        for (int f = 0; f < NFC; ++f) {
            if (f >= n8) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int n = 8 * f + 2 * tt + h;
                if (n >= np || x >= rows) continue;
                double* dst = out + x + (long)n * ldo;
                if (EVEN) {
                    *reinterpret_cast<double2*>(dst) = make_double2(acc[0][f][h], acc[1][f][h]);
                } else {
                    dst[0] = acc[0][f][h];
                    if (x + 1 < rows) dst[1] = acc[1][f][h];
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <int RC>
static void launch_class(const DevTree<double>& t, const int64_t* items, long n, bool keep, cudaStream_t st) {
    if (n <= 0) return;
    using SM = SmallSmem<RC>;
    if (t.r % 2 == 0) k_finest_small<RC, true><<<(unsigned)n, SM::NT, sizeof(SM), st>>>(t, items, keep ? 1 : 0);
    else k_finest_small<RC, false><<<(unsigned)n, SM::NT, sizeof(SM), st>>>(t, items, keep ? 1 : 0);
}

int launch_finest_small(const Geom& g, const DevTree<double>& t, bool keep, cudaStream_t st) {
    if (t.n_fin_items == 0) return 0;
    int wpr = 8;
    while (wpr > 1 && t.n_fin * wpr > 148L * 64) wpr /= 2;
    const long blocks = (t.n_fin * wpr + 7) / 8;
    const unsigned grid = (unsigned)(blocks < 148L * 32 ? blocks : 148L * 32);
    with_cov_kind(cov_kind(g, true), [&](auto k) { k_cov_group<decltype(k)::value><<<grid, 256, 0, st>>>(g, t, wpr); });
    // largest class first
    const long n64 = t.n_fin_class[0], n32 = t.n_fin_class[1], n16 = t.n_fin_class[2];
    launch_class<64>(t, t.fin_items, n64, keep, st);
    launch_class<32>(t, t.fin_items + n64, n32, keep, st);
    launch_class<16>(t, t.fin_items + n64 + n32, n16, keep, st);
    return 1 + (n64 > 0) + (n32 > 0) + (n16 > 0);
}

template <int RC>
static cudaError_t prepare_class() {
    const int bytes = (int)sizeof(SmallSmem<RC>);
    cudaError_t e = cudaFuncSetAttribute((const void*)k_finest_small<RC, true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute((const void*)k_finest_small<RC, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 bytes);
    return e;
}

cudaError_t prepare_finest_small() {
    cudaError_t e = prepare_class<16>();
    if (e == cudaSuccess) e = prepare_class<32>();
    if (e == cudaSuccess) e = prepare_class<64>();
    return e;
}

}  // namespace mra
