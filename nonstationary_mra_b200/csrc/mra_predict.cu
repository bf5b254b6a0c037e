// Prediction (FP64, r <= 64; ...-prior.cpp:271-392, class_approximation-predict.cpp:
// 105-189), in launches split by what is independent.  One CTA per level M-2 region
// did all of it, a handful of points wide: 4.2 of the 20 ms of predicting 16,384 points
// from 262,144 clustered observations (r = 64, eight levels); 1.9 ms as
//   k_cov_set, k_condition_set  (mra_finest.cu) V and U of the points against their
//                       ancestors, in chunks of at most 64 points below one level M-3
//                       region: 0.5 ms
//   k_predict_region    the part of a finest region's own observations:
//                       Pc = L_Sigma^{-1} (C - U_S^T U_P), V -= B^ Pc; a few points
//                       per region, so streams of U_S and B^ against vectors: 0.8 ms
//                       (k_predict_tiles: more than kPredVector of them)
//   k_predict_back      from the deepest ancestor up: K = L~_j^{-1} V_j,
//                       V_{0..j-1} -= G_j^T K, and the points' sums, in the same
//                       chunks: 0.6 ms (1.06 with the products of all eight column
//                       fragments in one unrolled body and the narrow ones skipped)
#include <algorithm>

#include "mra_cond.cuh"

namespace mra {

constexpr int kPredBatch = 4;   // points of a finest region taken together

// variance and mean of point p from its column c of Pc; one warp
__device__ __forceinline__ void region_sums(const DevTree<double>& t, const double* c, long o0, int n, long p) {
    const int lane = threadIdx.x & 31;
    double ss = 0.0, mm = 0.0;
    for (int o = lane; o < n; o += 32) {
        ss = fma(c[o], c[o], ss);
        mm = fma(c[o], t.yt[o0 + o], mm);
    }
    for (int d = 16; d > 0; d >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, d);
        mm += __shfl_xor_sync(0xffffffffu, mm, d);
    }
    if (lane == 0) {
        t.var[p] = -ss;
        t.mean[p] = mm;
    }
}

// At most kPredVector points of a region: the kernel reads U_S, L_Sigma and B^ once per
// kPredBatch points and is bound by the latency of its short phases (16 observations
// and one or two points per region are typical), so by the regions in flight: four CTAs
// per SM, the factor in blocks of 32 rows, one row per lane (two CTAs of twice the
// shared memory, blocks of 64 rows: 1.44 ms at the size above, this 0.8).
template <int KIND>
__global__ void __launch_bounds__(kThreads, 4) k_predict_region(Geom g, DevTree<double> t) {
    constexpr int PB = kPredBatch;
    __shared__ __align__(16) double stage[7 * kCovChunk];
    __shared__ double Lb[32 * 33], iv[32], xs[PB * 32];
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    double* Ps = reinterpret_cast<double*>(la_dyn_smem);  // [PB][Lr]: U_P; then [PB][256]: Pc
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int Lr = t.L * t.r;
    const FinChunk ch = t.pitems[blockIdx.x];
    const long k = ch.unit, pk = ch.lo, o0 = t.obs_off[k];
    const int npk = ch.n, n = (int)(t.obs_off[k + 1] - o0);
    if (n == 0) {
        for (int q = tid; q < npk; q += kThreads) t.mean[pk + q] = t.var[pk + q] = 0.0;
        return;
    }
    double* Pc = t.Pc + t.pc_off[k] + (pk - t.pred_off[k]) * n;  // n x npk
    const double* Ls = t.Lsig + t.lsig_off[k];
    cov_block<double, KIND>(g, t.pts, t.obs0 + o0, n, t.pred0 + pk, npk, false, Pc, n, stage);
    for (int p0 = 0; p0 < npk; p0 += PB) {
        const int np = min(PB, npk - p0);
        __syncthreads();
#pragma unroll
        for (int p = 0; p < PB; ++p)
            for (int x = tid; x < Lr; x += kThreads) Ps[p * Lr + x] = p < np ? t.P[(pk + p0 + p) * Lr + x] : 0.0;
        __syncthreads();
        // Pc = C - U_S^T U_P, one warp per observation
        for (int o = w; o < n; o += kThreads / 32) {
            const double* u = t.Ufin + (o0 + o) * Lr;
            double s[PB] = {};
#pragma unroll 8
            for (int x = lane; x < Lr; x += 32) {
                const double v = u[x];
#pragma unroll
                for (int p = 0; p < PB; ++p)
                    if (p < np) s[p] = fma(v, Ps[p * Lr + x], s[p]);
            }
#pragma unroll
            for (int p = 0; p < PB; ++p) {
                if (p >= np) break;
                for (int d = 16; d > 0; d >>= 1) s[p] += __shfl_xor_sync(0xffffffffu, s[p], d);
                if (lane == p) Pc[o + (long)(p0 + p) * n] -= s[p];
            }
        }
        // Pc <- L_Sigma^{-1} Pc in blocks of 32 rows: warp p solves point p, then all rows below
        for (int b0 = 0; b0 < n; b0 += 32) {
            const int nb = min(32, n - b0);
            for (int e = tid; e < nb * 32; e += kThreads) {
                const int i = e & 31, j = e >> 5;
                if (i < nb) {
                    const double v = Ls[(b0 + i) + (long)(b0 + j) * n];
                    Lb[i + j * 33] = v;
                    if (i == j) iv[i] = 1.0 / v;
                }
            }
            __syncthreads();
            if (w < np) {
                double* c = Pc + b0 + (long)(p0 + w) * n;
                double x = lane < nb ? c[lane] : 0.0;
                for (int j = 0; j < nb; ++j) {
                    const double xj = __shfl_sync(0xffffffffu, x, j) * iv[j];
                    if (lane == j) x = xj;
                    if (lane > j && lane < nb) x = fma(-Lb[lane + j * 33], xj, x);
                }
                xs[w * 32 + lane] = x;
                if (lane < nb) c[lane] = x;
            }
            __syncthreads();
            if (b0 + 32 >= n) break;
            for (int i = b0 + 32 + tid; i < n; i += kThreads) {
                double s[PB] = {};
#pragma unroll 8
                for (int j = 0; j < 32; ++j) {
                    const double v = Ls[i + (long)(b0 + j) * n];
#pragma unroll
                    for (int p = 0; p < PB; ++p)
                        if (p < np) s[p] = fma(v, xs[p * 32 + j], s[p]);
                }
#pragma unroll
                for (int p = 0; p < PB; ++p)
                    if (p < np) Pc[i + (long)(p0 + p) * n] -= s[p];
            }
            __syncthreads();
        }
        if (w < np) region_sums(t, Pc + (long)(p0 + w) * n, o0, n, pk + p0 + w);
        // V -= B^ Pc
        for (int c0 = 0; c0 < n; c0 += 256) {
            const int nc = min(256, n - c0);
            __syncthreads();
            if (tid < nc) {
#pragma unroll
                for (int p = 0; p < PB; ++p)
                    if (p < np) Ps[p * 256 + tid] = Pc[c0 + tid + (long)(p0 + p) * n];
            }
            __syncthreads();
            for (int x = tid; x < Lr; x += kThreads) {
                const double* b = t.Bhat + (o0 + c0) * Lr + x;
                double s[PB] = {};
#pragma unroll 8
                for (int o = 0; o < nc; ++o) {
                    const double v = b[(long)o * Lr];
#pragma unroll
                    for (int p = 0; p < PB; ++p)
                        if (p < np) s[p] = fma(v, Ps[p * 256 + o], s[p]);
                }
#pragma unroll
                for (int p = 0; p < PB; ++p)
                    if (p < np) t.Bt[(pk + p0 + p) * Lr + x] -= s[p];
            }
        }
    }
}

// More points: tile products, which read the region's blocks once per 64 points.
__global__ void __launch_bounds__(kThreads, 2) k_predict_tiles(Geom g, DevTree<double> t) {
    LaSmem<double>& sm = la_smem<double>();
    const int Lr = t.L * t.r;
    const FinChunk ch = t.pitems[t.n_pvec + blockIdx.x];
    const long k = ch.unit, pk = ch.lo, o0 = t.obs_off[k];
    const int npk = ch.n, n = (int)(t.obs_off[k + 1] - o0);
    if (n == 0) {
        for (int q = threadIdx.x; q < npk; q += kThreads) t.mean[pk + q] = t.var[pk + q] = 0.0;
        return;
    }
    double* Pc = t.Pc + t.pc_off[k] + (pk - t.pred_off[k]) * n;  // n x npk
    fill_cov<double>(g, t.pts, t.obs0 + o0, n, t.pred0 + pk, npk, false, Pc, n, sm);
    __syncthreads();
    gemm<double, true, false>(n, npk, Lr, -1.0, t.Ufin + o0 * Lr, Lr, t.P + pk * Lr, Lr, 1.0, Pc, n, sm);
    trsm_left_lower<double>(n, npk, t.Lsig + t.lsig_off[k], n, Pc, n, sm);
    for (int q = threadIdx.x >> 5; q < npk; q += kThreads / 32) region_sums(t, Pc + (long)q * n, o0, n, pk + q);
    gemm<double, false, false>(Lr, npk, n, -1.0, t.Bhat + o0 * Lr, Lr, Pc, n, 1.0, t.Bt + pk * Lr, Lr, sm);
}

template <int RC>
struct BackSmem {
    CondSmem<RC> c;
    double mean[64], var[64];
};

// acc -= G_j^T K over slab q, F column fragments; K [column][row] where Cond keeps V
template <class CC, int F>
__device__ __forceinline__ void back_slab(const CC& cond, double (&acc)[2][CC::NF][2], const double* A, int q) {
    const int sw = cond_swz(cond.g), RC = 16 * CC::RW;
    const double* a0 = A + (16 * cond.wr + cond.g) * TK64;
#pragma unroll 1
    for (int s = 0; s < CC::KN / 8; ++s) {
        const int offa = ((4 * s + cond.t) ^ sw) * 2, offb = offa + q * TK64;
        const double2 x0 = neg2(lds2(a0 + offa)), x1 = neg2(lds2(a0 + 8 * TK64 + offa));
        double2 y[F];
#pragma unroll
        for (int f = 0; f < F; ++f) {
            const int c = (f * CC::CW + cond.wc) * 8;
            y[f] = lds2(cond.sm.B[c / CC::VC] + (c % CC::VC + cond.g) * RC + offb);
        }
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

template <int RC, bool EVEN>
__global__ void __launch_bounds__(kCondThreads, CondSmem<RC>::CTAS) k_predict_back(DevTree<double> t, CondSet set) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    using CC = Cond<RC, EVEN>;
    BackSmem<RC>& bs = *reinterpret_cast<BackSmem<RC>*>(la_dyn_smem);
    CondSmem<RC>& sm = bs.c;
    const int r = t.r, L = t.L, m = t.M - 2;
    const long rr = (long)r * r, Lr = (long)L * r;
    const FinChunk ch = set.chunks[blockIdx.x];
    const long unit = ch.unit;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    CC cond(sm, r);
    const int g = cond.g, tt = cond.t, wr = cond.wr, wc = cond.wc;
    // prior variance and the sums of U_P
    for (int q = w; q < ch.n; q += kCondThreads / 32) {
        const double* u = set.U + (ch.lo + q) * Lr;
        double ss = 0.0;
        for (int x = lane; x < Lr; x += 32) ss = fma(u[x], u[x], ss);
        for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
        if (lane == 0) {
            const long ip = set.pt0 + ch.lo + q;
            bs.var[q] = t.pts.s2[ip] + t.pts.t2[ip] - ss + t.var[ch.lo + q];
            bs.mean[q] = t.mean[ch.lo + q];
        }
    }
    const int ng = m > 0 ? t.J : 1;
    const long g0 = m > 0 ? unit * t.J : 0;
    // level M-2 per sibling group, then the shared ancestors upwards
    for (int s = 0; s < ng + m; ++s) {
        const int j = s < ng ? m : m - 1 - (s - ng);
        long a, lo = ch.lo, hi = ch.lo + ch.n;
        if (s < ng) {
            a = t.lstart[m] + g0 + s;
            if (set.glo[g0 + s] > lo) lo = set.glo[g0 + s];
            if (set.ghi[g0 + s] < hi) hi = set.ghi[g0 + s];
            if (lo >= hi) continue;
        } else {
            a = ancestor(t, m - 1, unit, j);
        }
        const int N = (int)(hi - lo), N8 = (N + 7) & ~7, q0 = (int)(lo - ch.lo);
        double* V = set.V + lo * Lr;
        const int nf = cond.frags(N);
        const double* P = t.Lpinv + a * rr;
        __syncthreads();  // the previous step is done with the shared memory
        cond.load_inv(P, 0, sm.A[0]);
        if (CC::NP > 1) cond.load_inv(P, 1, sm.A[1]);
        constexpr int PV = EVEN ? RC / 2 : RC;  // copies per column
        for (int e = tid; e < N8 * PV; e += kCondThreads) {  // V_j as [column][row]
            const int c = e / PV, x = (EVEN ? 2 : 1) * (e % PV);
            const bool ok = c < N && x < r;
            double* dst = sm.B[c / CC::VC] + (c % CC::VC) * RC + (((x >> 1) ^ cond_swz(c)) << 1) + (x & 1);
            const double* src = ok ? V + (long)c * Lr + (long)j * r + x : V;
            if (EVEN) cp_async16z(dst, src, ok);
            else cp_async8(dst, src, ok);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        double acc[2][CC::NF][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int f = 0; f < CC::NF; ++f) acc[i][f][0] = acc[i][f][1] = 0.0;
        const int end = (16 * (wr + 1) < r ? 16 * (wr + 1) : r + 7) / 8;
        const int nk = 16 * wr < r ? nf : 0;
        cond.mma_inv_n(nk, acc, sm.A[0], 0, end < CC::KN / 8 ? end : CC::KN / 8);
        if (CC::NP > 1 && end > TK64 / 8) cond.mma_inv_n(nk, acc, sm.A[1], 1, end - TK64 / 8);
        __syncthreads();
        // K = L~^{-1} V_j in V_j's place; G_j's first slab on its way
        const double* G = t.G + t.u_off[j] + (a - t.lstart[j]) * (long)j * rr;
        const int ns = (r + TK64 - 1) / TK64, jr = j * r, nv = (jr + RC - 1) / RC * ns;
        auto issue = [&](int v) {  // slab v % ns of row tile v / ns
            if (v < nv) {
                const int x0 = v / ns * RC;
                cond.load_rows(sm.A[v & 1], G + (long)x0 * r, r, min(RC, jr - x0), RC, v % ns * TK64, r);
            }
            cp_async_commit();
        };
        issue(0);
#pragma unroll
        for (int f = 0; f < CC::NF; ++f) {
            const int c = (f * CC::CW + wc) * 8 + 2 * tt;
            if (f >= nk) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<double2*>(sm.B[c / CC::VC] + (c % CC::VC + h) * RC +
                                            (((8 * wr + g) ^ cond_swz(2 * tt + h)) << 1)) =
                    make_double2(acc[0][f][h], acc[1][f][h]);
        }
        __syncthreads();
        {
            const double* v = t.vpost + a * r;
            for (int q = w; q < N; q += kCondThreads / 32) {
                const double* col = sm.B[q / CC::VC] + (q % CC::VC) * RC;
                double ss = 0.0, mm = 0.0;
                for (int x = lane; x < r; x += 32) {
                    const double c = col[(((x >> 1) ^ cond_swz(q)) << 1) + (x & 1)];
                    ss = fma(c, c, ss);
                    mm = fma(c, v[x], mm);
                }
                for (int d = 16; d > 0; d >>= 1) {
                    ss += __shfl_xor_sync(0xffffffffu, ss, d);
                    mm += __shfl_xor_sync(0xffffffffu, mm, d);
                }
                if (lane == 0) {
                    bs.var[q0 + q] += ss;
                    bs.mean[q0 + q] += mm;
                }
            }
        }
        // V_{0..j-1} -= G_j^T K
        for (int v = 0; v < nv; ++v) {
            const int x0 = v / ns * RC, q = v % ns, rows = min(RC, jr - x0);
            const bool on = 16 * wr < rows;
            if (q == 0) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int x = 16 * wr + 8 * i + g;
#pragma unroll
                    for (int f = 0; f < CC::NF; ++f) {
                        if (f >= nf) continue;
                        const int c = (f * CC::CW + wc) * 8 + 2 * tt;
#pragma unroll
                        for (int h = 0; h < 2; ++h) acc[i][f][h] = (x < rows && c + h < N) ? V[x0 + x + (long)(c + h) * Lr] : 0.0;
                    }
                }
            }
            cp_async_wait<0>();
            __syncthreads();
            issue(v + 1);
            if (on) {
                const double* A = sm.A[v & 1];
                // widths as in Cond::mma_slab_n
                if (nf == 1) back_slab<CC, 1>(cond, acc, A, q);
                else if (nf == 2) back_slab<CC, 2>(cond, acc, A, q);
                else if constexpr (CC::NF > 2) {
                    if (nf > 6) { if constexpr (CC::NF >= 8) back_slab<CC, 8>(cond, acc, A, q); }
                    else if (nf > 4) { if constexpr (CC::NF >= 6) back_slab<CC, 6>(cond, acc, A, q); }
                    else if (nf > 2) back_slab<CC, 4>(cond, acc, A, q);
                }
            }
            if (q == ns - 1) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int x = 16 * wr + 8 * i + g;
#pragma unroll
                    for (int f = 0; f < CC::NF; ++f) {
                        if (f >= nf) continue;
                        const int c = (f * CC::CW + wc) * 8 + 2 * tt;
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            if (x < rows && c + h < N) V[x0 + x + (long)(c + h) * Lr] = acc[i][f][h];
                    }
                }
            }
        }
    }
    __syncthreads();
    for (int q = tid; q < ch.n; q += kCondThreads) {
        t.mean[ch.lo + q] = bs.mean[q];
        t.var[ch.lo + q] = bs.var[q];
    }
}

template <int RC>
static void launch_back(const DevTree<double>& t, const CondSet& s, cudaStream_t st) {
    if (t.r % 2 == 0) k_predict_back<RC, true><<<(unsigned)s.n, kCondThreads, sizeof(BackSmem<RC>), st>>>(t, s);
    else k_predict_back<RC, false><<<(unsigned)s.n, kCondThreads, sizeof(BackSmem<RC>), st>>>(t, s);
}

int launch_predict_chunks(const Geom& g, const DevTree<double>& t, cudaStream_t st) {
    const CondSet s{t.pchunks, t.n_pchunks, t.pred0, t.Bt, t.P, t.pglo, t.pghi};
    int launches = launch_condition_set(g, t, s, st);
    if (t.n_pvec > 0) {
        const size_t sb = kPredBatch * (size_t)std::max(t.L * t.r, 256) * sizeof(double);
        with_cov_kind(cov_kind(g, true), [&](auto k) {
            k_predict_region<decltype(k)::value><<<(unsigned)t.n_pvec, kThreads, sb, st>>>(g, t);
        });
        ++launches;
    }
    if (t.n_pitems > t.n_pvec) {
        k_predict_tiles<<<(unsigned)(t.n_pitems - t.n_pvec), kThreads, sizeof(LaSmem<double>), st>>>(g, t);
        ++launches;
    }
    if (t.r <= 16) launch_back<16>(t, s, st);
    else if (t.r <= 32) launch_back<32>(t, s, st);
    else launch_back<64>(t, s, st);
    return launches + 1;
}

template <int RC>
static cudaError_t prepare_back() {
    cudaError_t e = cudaSuccess;
    for (const void* fn : {(const void*)k_predict_back<RC, true>, (const void*)k_predict_back<RC, false>})
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BackSmem<RC>));
    return e;
}

cudaError_t prepare_predict() {
    cudaError_t e = cudaFuncSetAttribute((const void*)k_predict_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(LaSmem<double>));
    if (e == cudaSuccess) e = prepare_back<16>();
    if (e == cudaSuccess) e = prepare_back<32>();
    if (e == cudaSuccess) e = prepare_back<64>();
    return e;
}

cudaError_t set_gemm_tiles_predict(const int nw[3]) { return cudaMemcpyToSymbol(c_gemm_nw, nw, 3 * sizeof(int)); }

}  // namespace mra
