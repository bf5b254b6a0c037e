// Region kernels of the MRA hot path, templated on the storage type T
// (double: plain FP64 path; float: mixed path, FP32 storage and 3xTF32 tensor
// products, FP64 diagonal blocks and log-likelihood accumulation).
//
// Schedule of one log-likelihood (one launch per stage and tree level):
//   k_fields            sigma^2/beta/tau^2 at every knot, observation and
//                       prediction point (class_nonstationary_covariance.cpp:479-573)
//   (mra_prior.cu)      prior, levels 0..M-2: U_{i,j} = L_{a_j}^{-1} V_j,
//                       L_i = chol(K_i)   (class_approximation.cpp:46-50,84-169)
//   (mra_finest.cu)     finest level: conditioning, Sigma, L_Sigma, y~, B^ and
//                       the log-lik terms
//                       (...-loop-regions-at-finest-level-in-prior.cpp:90-269)
//   (mra_posterior.cu)  posterior, levels M-2..0 (...-posterior-inference.cpp:14-265,
//                       class_approximation.cpp:186-306)
//   k_reduce            deterministic sum of the per-region terms
//   (mra_predict.cu)    prediction; k_predict for FP32 storage and r > 64, one CTA
//                       per level M-2 region (its finest children's predictions
//                       together)
//                       (...-prior.cpp:271-392, class_approximation-predict.cpp:105-189)
#include "mra_kernels.cuh"

namespace mra {

// ---------------------------------------------------------------------------
// a1: fields
// ---------------------------------------------------------------------------
// One thread per point and field (blockIdx.y): a point's basis sums are chains of
// an exponential or a polynomial per basis function, so the three fields run side
// by side, in small blocks that spread over the chip (8,192 points with two fields
// of 9 functions: 11.2 us with one thread per point in blocks of 256, 8.5 us now).
constexpr int kFieldThreads = 64;

__device__ __forceinline__ double field_value(const Geom& g, const FieldParams& fp, int f, const Pt& p) {
    const double* th = fp.theta;
    if (!g.nonstat) return th[6 + f];
    double v = th[3 + f];
    const long nb = fp.nb[f];
    const double* c = fp.centers[f];
    const double* w = fp.weights[f];
#pragma unroll 3
    for (long b = 0; b < nb; ++b) {
        const Pt q{c[b], c[nb + b], c[2 * nb + b]};
        const double d = point_distance(g, p, q) / fp.basis_len;
        if (fp.basis == 0) {
            const double u = 1 - d, u2 = u * u;
            const double phi = u2 * u2 * u2 * (35 * d * d + 18 * d + 3) * w[b] / 3;
            v += d >= 1 ? 0.0 : phi;
        } else {
            v += exp(-0.5 * d * d) * w[b];
        }
    }
    return th[f] * exp(v);
}

__device__ __forceinline__ void store_field(int f, long i, double v, double* s2, double* beta, double* t2, double* ss) {
    if (f == 0) {
        s2[i] = v;
        ss[i] = sqrt(fabs(v));  // the products sigma_a sigma_b are of one sign, that of the scale
    } else {
        (f == 1 ? beta : t2)[i] = v;
    }
}

__global__ void __launch_bounds__(kFieldThreads)
    k_fields(Geom g, FieldParams fp, const double* __restrict__ c0, const double* __restrict__ c1,
             const double* __restrict__ c2, long n, double* __restrict__ s2, double* __restrict__ beta,
             double* __restrict__ t2, double* __restrict__ ss) {
    const long i = (long)blockIdx.x * kFieldThreads + threadIdx.x;
    if (i >= n) return;
    const int f = blockIdx.y;
    store_field(f, i, field_value(g, fp, f, Pt{c0[i], c1[i], c2[i]}), s2, beta, t2, ss);
}

// The same for the points p2 [3][n2] then p1 [3][n1] with the parameters passed by
// value (small models: nothing to copy first); also gathers the coordinates.
__global__ void __launch_bounds__(kFieldThreads)
    k_fields_inline(Geom g, FieldParams fp, const __grid_constant__ InlineTables tab, const double* __restrict__ p2,
                    long n2, const double* __restrict__ p1, long n1, PointBuffers o) {
    const long i = (long)blockIdx.x * kFieldThreads + threadIdx.x;
    if (i >= n1 + n2) return;
    const int f = blockIdx.y;
    const double* src = i < n2 ? p2 + i : p1 + (i - n2);
    const long n = i < n2 ? n2 : n1;
    const Pt p{src[0], src[n], src[2 * n]};
    long off = 0;
    fp.theta = tab.theta;
    for (int q = 0; q < 3; ++q) {
        fp.centers[q] = tab.v + off;
        fp.weights[q] = tab.v + off + 3 * fp.nb[q];
        off += 4 * fp.nb[q];
    }
    if (f == 0) {
        o.c[0][i] = p.c0;
        o.c[1][i] = p.c1;
        o.c[2][i] = p.c2;
    }
    store_field(f, i, field_value(g, fp, f, p), o.f[0], o.f[1], o.f[2], o.f[3]);
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
            trsm_left_lower<T>(r, np, t.Lpost + a * rr, r, KcB, Lr, sm);
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
// Straight-line nonstationary forms: tiles of RT rows x CT columns by the blocks of
// mra_device.cuh (4001 x 3003 planar entries: 62 to 64 us a call, 1.5 TB/s of results; by the
// entry-per-thread kernel below 142 to 144).  Two CTAs per SM, whose 128 registers hold the
// entry without spills: 3 take 64 and 66 us, 4 take 66 and 68.
template <int KIND>
__global__ void __launch_bounds__(kCovThreads, 2) k_cov_tiles(CovScale scale, PointSet P, long a0, int na, long b0, int nb,
                                                              int self, int RT, int CT, double* out) {
    __shared__ __align__(16) double stage[7 * kCovChunk];
    const int t0 = blockIdx.x * RT, q0 = blockIdx.y * CT;
    const int nr = min(RT, na - t0), nc = min(CT, nb - q0);
    using F = CovForm<KIND>;
    cov_block_fast<double, F::NU, F::PREF, true>(P, a0 + t0, nr, b0 + q0, nc, self != 0, t0 - q0,
                                                      out + t0 + (long)q0 * na, na, scale, stage);
}

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
                   long n, double* s2, double* beta, double* t2, double* ss, cudaStream_t st) {
    if (n <= 0) return;
    const dim3 grid((unsigned)((n + kFieldThreads - 1) / kFieldThreads), 3);
    k_fields<<<grid, kFieldThreads, 0, st>>>(g, fp, c0, c1, c2, n, s2, beta, t2, ss);
}
void launch_fields_inline(const Geom& g, const FieldParams& fp, const InlineTables& tab, const double* p2, long n2,
                          const double* p1, long n1, const PointBuffers& o, cudaStream_t st) {
    const long n = n1 + n2;
    if (n <= 0) return;
    const dim3 grid((unsigned)((n + kFieldThreads - 1) / kFieldThreads), 3);
    k_fields_inline<<<grid, kFieldThreads, 0, st>>>(g, fp, tab, p2, n2, p1, n1, o);
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
    const int kind = g.dist_scale >= 0 ? cov_kind(g, true) : 0;  // exp_neg takes no negative exponent
    if (kind > 0) {
        // long column runs, unless that leaves the chip short of blocks
        int RT = 256, CT = kCovChunk;
        while ((long)((na + RT - 1) / RT) * ((nb + CT - 1) / CT) < 4 * 148 && CT > 8) RT > 64 ? RT /= 2 : CT /= 2;
        const long gy = (nb + CT - 1) / CT;
        if (gy <= 65535) {
            const dim3 grid((unsigned)((na + RT - 1) / RT), (unsigned)gy);
            // the product with the rounded root that matern() multiplies by, itself not rounded
            const long double f = (g.nu_x2 == 3 ? (long double)1.7320508075688772 : 1.0L) * g.dist_scale;
            const CovScale scale{g.dist_scale, (double)f, (double)(f - (double)f)};
            with_cov_kind(kind, [&](auto k) {
                if constexpr (decltype(k)::value > 0)
                    k_cov_tiles<decltype(k)::value><<<grid, kCovThreads, 0, st>>>(scale, P, a0, na, b0, nb, self ? 1 : 0, RT,
                                                                                  CT, out);
            });
            return;
        }
    }
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
    set((const void*)k_predict<T>);
    set((const void*)k_reduce<T>);
    set((const void*)k_sample<T>);
    return e;
}

// every file with FP64 products holds its own copy of the widths
cudaError_t set_gemm_tiles(const int nw[3]) {
    cudaError_t e = cudaMemcpyToSymbol(c_gemm_nw, nw, 3 * sizeof(int));
    for (auto set : {set_gemm_tiles_prior, set_gemm_tiles_posterior, set_gemm_tiles_predict})
        if (e == cudaSuccess) e = set(nw);
    return e;
}

cudaError_t prepare_kernels() {
    cudaError_t e = prepare_type<double>();
    if (e == cudaSuccess) e = prepare_type<float>();
    if (e == cudaSuccess) e = prepare_prior();
    if (e == cudaSuccess) e = prepare_predict();
    if (e == cudaSuccess) e = prepare_posterior();
    return e == cudaSuccess ? prepare_finest() : e;
}

#define MRA_INSTANTIATE(T)                                                                                   \
    template void launch_predict<T>(const Geom&, const DevTree<T>&, int, cudaStream_t);                     \
    template void launch_reduce<T>(const DevTree<T>&, double*, cudaStream_t);                               \
    template void launch_sample<T>(const DevTree<T>&, const double*, const double*, double*, int, cudaStream_t);
MRA_INSTANTIATE(double)
MRA_INSTANTIATE(float)

}  // namespace mra
