// Launch interface between the C-ABI layer (mra_api.cu) and the region
// kernels (mra_kernels.cu), templated on the storage type T (double: plain
// FP64 path, float: mixed path).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/mra_b200.h"
#include "mra_device.cuh"

namespace mra {

// A run of observations that share their ancestors of levels 0..M-3 (unit: the
// local index of the level M-3 region, 0 when M = 2), conditioned by one CTA.
struct FinChunk {
    int64_t lo;
    int32_t n;
    int32_t unit;
};
// A finest region of at most kFinTile observations is one work item; a sibling
// group is one item when its children hold at most kChildMax and together at
// most kGroupMax observations (FP64).
constexpr int kFinTile = 64, kGroupMax = 64, kChildMax = 32;
struct HeavyTile {
    int32_t h;       // index into DevTree::heavy
    uint16_t bi, bj; // 64 x 64 tile of Sigma, bi >= bj
};

// Everything a kernel needs to address the resident structure and buffers.
template <typename T>
struct DevTree {
    int J, M, r, L;            // L = M-1 ancestor levels of a finest region
    int lj;                    // log2 J
    int lstart[kMaxLevels];    // first region of each interior level
    long n_int, n_fin, n_obs, n_pred;
    long obs0, pred0;          // first obs / pred index in the joint point arrays
    int tf;                    // largest subtree (in observations) kept in factored form
    PointSet pts;              // knots | obs | preds, with their fields (FP64)
    const double* y;           // [n_obs]
    const int64_t* obs_off;    // [n_fin+1]
    const int64_t* pred_off;   // [n_fin+1]
    const int64_t* fin_anc;    // [n_fin][L] ancestors of each finest region, level 0 first
    const int64_t* sub_lo;     // [n_int] first observation of each interior region's subtree
    const int64_t* sub_hi;     // [n_int] one past the last
    const int64_t* child_lo;   // [J^(M-2)] first finest child of each level M-2 region
    const int64_t* child_hi;   // one past the last
    const FinChunk* chunks;    // [n_chunks] runs of observations conditioned together
    long n_chunks;
    const int64_t* fin_items;  // [n_fin_items] small finest regions: a value v < J^(M-2) is the sibling group v,
                               // else the finest region v - J^(M-2); FP64: by tile class (64, 32, 16), each most
                               // expensive first
    long n_fin_items, n_fin_class[3];
    const int64_t* heavy;      // [n_heavy] finest regions of more than 64 observations (FP64), largest first
    long n_heavy;
    const HeavyTile* heavy_tiles;  // [n_heavy_tiles] lower tiles of their Sigma
    long n_heavy_tiles;
    const int64_t* pred_order; // [J^(M-2)] level M-2 regions (local index), most expensive prediction work first
    const int64_t* post_order; // [n_int] per level m, at level_start(m): the level's regions (local index), its
                               // n_dense[m] dense ones first, each kind most expensive step first
    long n_dense[kMaxLevels];
    long n_mid[kMaxLevels];    // of its factored ones, those of more than 64 rows (they come first)
    long n_fused;              // last factored regions of level M-2 in post_order whose posterior (outside
                               // prediction) comes with their finest group
    const FinChunk* pchunks;   // [n_pchunks] runs of prediction points conditioned together (FP64, r <= 64)
    long n_pchunks;
    const int64_t* pglo;       // [J^(M-2)] first prediction point of each level M-2 region
    const int64_t* pghi;       // one past the last
    const FinChunk* pitems;    // [n_pitems] runs of prediction points of one finest region: the n_pvec of at most
                               // kPredVector points first, most expensive first
    long n_pitems, n_pvec;
    const int8_t* factored;    // [n_int] 1: the region's posterior output is kept as F, f
    const int8_t* active;      // [n_int] sub-tree sharding: 0 = the region belongs to another rank's
                               // sub-tree and is skipped; nullptr: every region is computed
    const int64_t* dslot;      // [n_int] slot of a dense region among its level's dense regions (-1: factored)
    const int64_t* lsig_off;   // [n_fin+1] offsets of the n_k x n_k blocks
    const int64_t* pc_off;     // [n_fin+1] offsets of the n_k x n_p,k prediction blocks
    int64_t u_off[kMaxLevels]; // offset of level m's U (= G) blocks, m*r*r per region
    // prior
    T* Lprior;                 // [n_int][r*r]
    T* Pinv;                   // [n_int][r*r] inverse of each prior factor (L^{-1} applied as a product)
    double* ldprior;           // [n_int] 2 sum log diag of the prior factor
    T* U;                      // per level m: [J^m][(m r) x r], ld = m r
    T* Ufin;                   // [n_obs][L r]   finest U_{k,j} columns, obs-major
    T* Bhat;                   // [n_obs][L r]   B^ transposed, obs-major (the finest F)
    double* yt;                // [n_obs]        L_Sigma^{-1} y (the finest f)
    T* Lsig;                   // CSR n_k x n_k  finest Cholesky factors
    // posterior
    T* Lpost;                  // [n_int][r*r]
    double* vpost;             // [n_int][r]
    T* G;                      // like U: [J^m][r x (m r)], ld = r (prediction mode)
    T* Lpinv;                  // [n_int][r*r] inverse of each posterior factor (FP64 prediction mode, r <= 64), else null
    double* dpost;             // [n_int] posterior log-lik terms
    double* dchild;            // [n_fin] log-lik terms of each finest region (or of the group it leads)
    double* dfin;              // [J^(M-2)] finest-level log-lik terms of each sibling group
    int fuse_post;             // 1: the finest stage ends with the level M-2 posterior
    double* heavy_inv;         // [n_heavy][64 x 64] inverse of the current diagonal tile
    T* aout[2];                // dense A~ slices of one level's dense regions (by dslot), ping-pong by level parity
    double* wout[2];           // dense w~ of one level's dense regions (by dslot)
    T* Fbuf[2];                // factored F of one level: [n_obs][m r]
    double* fbuf[2];           // factored f of one level: [n_obs]
    T* cbuf;                   // covariance blocks of a chunk of one prior level's regions; later the scratch of
                               // a chunk of one posterior level's dense regions
    long cbuf_elems;           // its size in elements
    T* ws;                     // per-CTA workspace (T)
    long ws_stride;
    double* wsd;               // per-CTA workspace (FP64)
    long wsd_stride;
    // prediction
    T* P;                      // [n_pred][L r]
    T* Bt;                     // [n_pred][L r]
    T* Pc;                     // CSR n_k x n_p,k
    double* mean;              // [n_pred]
    double* var;               // [n_pred]
    // bookkeeping
    int* queue;                // work-queue counters (kQueueCounters, zeroed before every evaluation):
                               // [0] small finest regions, [1] prediction items, [kQueuePost + m] posterior level m
    int* err;                  // [0]: status, [1]: region (low), [2]: region (high)
};

// Points conditioned on their ancestors: observations (V: B^, U: Ufin) or prediction
// points (V: Bt, U: P), L r entries per point.
template <typename T>
struct CondSetT {
    const FinChunk* chunks;
    long n;
    long pt0;             // first point in the joint point arrays
    T* V;
    T* U;
    const int64_t* glo;   // [J^(M-2)] points of each level M-2 region: first
    const int64_t* ghi;   // and one past the last
};
using CondSet = CondSetT<double>;

// Prediction points of a finest region handled as vectors, four per pass over its blocks; more go
// through tile products.  65,536 observations, 16 points per region, vectors / tiles: 1.11 / 0.94 ms
// with 64 observations per region, 2.26 / 2.48 with 16; 10 points: 1.55 / 1.73 with 16.
// The crossing lies lower where a region holds more observations (its blocks are read
// once per four points); the line is taken for the usual 16.
constexpr int kPredVector = 12;
constexpr int kQueuePost = 4;
constexpr int kQueueCounters = kQueuePost + kMaxLevels;

__host__ __device__ inline long level_start(int J, int m) {
    long s = 0, p = 1;
    for (int i = 0; i < m; ++i) { s += p; p *= J; }
    return s;
}
__host__ __device__ inline long level_count(int J, int m) {
    long p = 1;
    for (int i = 0; i < m; ++i) p *= J;
    return p;
}
__host__ __device__ inline long n_slices(int m) { return (long)m * (m + 1) / 2; }
template <typename T>
__device__ __forceinline__ bool skipped(const DevTree<T>& t, long region) {
    return t.active && !t.active[region];
}
// the region whose sub-tree holds a chunk: the level M-3 region (the root when M = 2)
template <typename T>
__device__ __forceinline__ long chunk_region(const DevTree<T>& t, long unit) {
    return t.M >= 3 ? t.lstart[t.M - 3] + unit : 0;
}
// the level-j ancestor of region `loc` (local index) of level m
template <typename T>
__device__ __forceinline__ long ancestor(const DevTree<T>& t, int m, long loc, int j) {
    return t.lstart[j] + (loc >> (t.lj * (m - j)));
}
// slice index of block (j,k), j <= k < m, row-major over the upper triangle
// (the order of class_approximation.cpp:62-73)
__host__ __device__ inline long slice_index(int m, int j, int k) { return (long)j * m - (long)j * (j - 1) / 2 + (k - j); }

__device__ inline void report_error(int* err, long region) {
    if (atomicCAS(&err[0], 0, 4 /* MRA_ERR_NOT_SPD */) == 0) {
        err[1] = (int)(region & 0x7fffffff);
        err[2] = (int)(region >> 31);
    }
}

// θ-dependent field evaluation parameters (device pointers)
struct FieldParams {
    int basis;                 // 0 Wendland, 1 Gaussian
    double basis_len;
    long nb[3];
    const double* centers[3];  // [3][nb]
    const double* theta;       // [0..2] scales, [3..5] intercepts, [6..8] stationary sill/range/nugget
    const double* weights[3];  // [nb]
};

// Sets the text returned by mra_last_error() on this thread.
void set_last_error(const char* msg);

// Validates a model description (kinds in range, positive basis length and
// non-NULL basis tables for nonstationary fields); sets the error text.
mra_status check_model(const mra_model* m);

// Opts the region kernels into their dynamic shared memory size on the current
// device; call before the first launch (and before any stream capture).
cudaError_t prepare_kernels();

// FP64 GEMM tile width per product-width bucket on the current device
// (c_gemm_nw in mra_device.cuh).
cudaError_t set_gemm_tiles(const int nw[3]);

void launch_fields(const Geom& g, const FieldParams& fp, const double* c0, const double* c1, const double* c2,
                   long n, double* s2, double* beta, double* t2, double* ss, cudaStream_t st);
// theta and the basis tables of a small model by value: per field the centers
// [3][nb] and the weights [nb], one after the other.
struct InlineTables {
    double theta[16];
    double v[432];
};
struct PointBuffers {
    double* c[3];
    double* f[4];  // sigma^2, beta, tau^2, sigma
};
void launch_fields_inline(const Geom& g, const FieldParams& fp, const InlineTables& tab, const double* p2, long n2,
                          const double* p1, long n1, const PointBuffers& o, cudaStream_t st);
// Events recorded around each covariance-block launch of a prior level, so
// that the caller can split the level's device time between the covariance
// launches and the region launches.
struct CovTiming {
    cudaEvent_t* ev;  // two per launch: before and after
    int cap;          // launches that can be timed
    int used;         // launches timed so far
    bool capturing;   // record as external nodes of the graph being captured
    bool overflow;    // a launch went untimed (cap reached)
};
// Covariance-block launches and region launches of one prior level, in chunks
// of regions whose blocks fit t.cbuf; returns the number of kernels launched.
template <typename T>
int launch_prior_level(const Geom& g, const DevTree<T>& t, int m, int grid, cudaStream_t st, CovTiming* tm = nullptr);
// Stream and events (timing disabled) for work beside the main stream's (heavy
// finest regions beside small ones, factored regions beside dense ones), and the
// number of observations of each heavy region (host memory, largest first).
struct Fork {
    cudaStream_t side;
    cudaEvent_t fork, join;
    const int* heavy_n;
};
// The finest level (without the level M-2 posterior); returns the number of kernels launched.
template <typename T>
int launch_finest(const Geom& g, const DevTree<T>& t, int grid, bool keep, cudaStream_t st, const Fork& fk);
// its small regions (FP64), with the posterior of groups taken whole unless `keep`
int launch_finest_small(const Geom& g, const DevTree<double>& t, bool keep, cudaStream_t st);
cudaError_t prepare_finest_small();
// covariance with the ancestors and conditioning of a set (r <= 64)
int launch_condition_set(const Geom& g, const DevTree<double>& t, const CondSet& s, cudaStream_t st);
// prediction in chunks (FP64, r <= 64); returns the number of kernels launched
int launch_predict_chunks(const Geom& g, const DevTree<double>& t, cudaStream_t st);
cudaError_t prepare_predict();
cudaError_t set_gemm_tiles_predict(const int nw[3]);
cudaError_t prepare_finest();
// One posterior level (FP64): its dense regions in chunks whose scratch fits
// t.cbuf, its factored ones beside them; returns the number of kernels launched, or -1
// (nothing launched) if the scratch does not hold one region of each kind.
int launch_posterior_level(const DevTree<double>& t, int m, int grid, bool keep, cudaStream_t st, const Fork& fk);
cudaError_t prepare_prior();
cudaError_t set_gemm_tiles_prior(const int nw[3]);
// sibling regions that one CTA of the prior takes together (their covariance
// blocks lie side by side): up to 64 columns, FP64 and r <= 64
inline int prior_batch(bool fp64, int r, int J) {
    const int sb = !fp64 || r > 64 ? 1 : (r <= 16 ? 4 : (r <= 32 ? 2 : 1));
    return sb < J ? sb : J;
}
cudaError_t prepare_posterior();
cudaError_t set_gemm_tiles_posterior(const int nw[3]);
// doubles of scratch of one dense region of level m: the slices (j, m), G and the inverse of L~
inline long dense_scratch(int m, int r) { return ((2L * m + 1) * r * r + 1) & ~1L; }
// of one factored region (tf rows at most): Y, S and R^{-1}; with `keep` also a dense region's
inline long fact_scratch(int m, int r, int tf, bool keep) {
    const long n = (long)r * tf + 2L * tf * tf, d = keep ? dense_scratch(m, r) : 0;
    const long e = n > d ? n : d;
    return e > 2 ? (e + 1) & ~1L : 2;
}
template <typename T>
void launch_predict(const Geom& g, const DevTree<T>& t, int grid, cudaStream_t st);
template <typename T>
void launch_reduce(const DevTree<T>& t, double* out, cudaStream_t st);
// out[i] = (To) in[i]
template <typename Ti, typename To>
void launch_convert(const Ti* in, To* out, long n, cudaStream_t st);
template <typename T>
void launch_sample(const DevTree<T>& t, const double* z_int, const double* z_obs, double* y_out, int grid,
                   cudaStream_t st);
void launch_cov_block(const Geom& g, const PointSet& P, long a0, int na, long b0, int nb, bool self, double* out,
                      cudaStream_t st);

}  // namespace mra
