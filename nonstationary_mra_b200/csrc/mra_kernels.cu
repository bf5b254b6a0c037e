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
//   k_predict           prediction, one CTA per level M-2 region (its finest
//                       children's predictions together)
//                       (...-prior.cpp:271-392, class_approximation-predict.cpp:105-189)
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
    set((const void*)k_predict<T>);
    set((const void*)k_reduce<T>);
    set((const void*)k_sample<T>);
    return e;
}

cudaError_t set_gemm_tiles(const int nw[3]) { return cudaMemcpyToSymbol(c_gemm_nw, nw, 3 * sizeof(int)); }

cudaError_t prepare_kernels() {
    cudaError_t e = prepare_type<double>();
    if (e == cudaSuccess) e = prepare_type<float>();
    if (e == cudaSuccess) e = prepare_prior();
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
