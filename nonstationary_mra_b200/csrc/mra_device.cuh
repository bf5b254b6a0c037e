// Device-side building blocks of the MRA hot path (sm_100a).
//
//  * covariance entries, following src/evaluate_covariance.cpp:155-313 and the
//    fields of src/class_nonstationary_covariance.cpp:479-573;
//  * CTA-cooperative dense primitives on column-major operands that may live
//    in global or shared memory, templated on the storage type T:
//      T = double  the plain FP64 path: products on the FP64 tensor pipe
//                  (mma.sync m8n8k4 f64);
//      T = float   the mixed path: operands stored in FP32, products on the
//                  tensor cores as three TF32 products (hi*hi + hi*lo + lo*hi,
//                  FP32-accurate) with FP32 accumulation.
//    Diagonal blocks of every Cholesky factorization and triangular solve are
//    computed in FP64 whatever T is, and log-determinants are accumulated in
//    FP64.  One CTA owns one region's problem; the region kernels in
//    mra_kernels.cu are sequences of these calls.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace mra {

constexpr int kThreads = 256;   // every region kernel runs 256-thread CTAs
constexpr int kMaxLevels = 16;  // NUM_LEVELS_M upper bound supported by the kernels

// ----------------------------------------------------------------------------
// geometry / covariance model (read-only per evaluation)
// ----------------------------------------------------------------------------
struct Geom {
    int nonstat;        // NONSTATIONARY_FLAG
    int distance;       // 0 chordal xyz, 1 great circle lon/lat degrees, 2 planar xy
    int nu_x2;          // 1: exponential, 3: Matern 3/2
    int pref_kind;      // 0: (x)^1.5, 1: (x)^1, 2: pow(x, pref_exp)
    double pref_exp;
    double dist_scale;
};

struct Pt {
    double c0, c1, c2;
};

// Models whose FP64 entries take the short forms: nonstationary, straight-line distance, prefactor
// exponent 1.5 or 1 (and a scale that is a number: exp_neg passes no undefined exponent on).
__host__ __device__ __forceinline__ bool fast_form(const Geom& g) {
    return g.nonstat && g.distance != 1 && g.pref_kind != 2 && g.dist_scale == g.dist_scale;
}

__device__ __forceinline__ double point_distance(const Geom& g, const Pt& a, const Pt& b) {
    if (g.distance == 1) {
        // great_circle_dist, evaluate_covariance.cpp:9-25
        const double k = 3.14159265358979323846 / 180.0;
        double lon1 = a.c0 * k, lon2 = b.c0 * k, lat1 = a.c1 * k, lat2 = b.c1 * k;
        double ang = sin(lat1) * sin(lat2) + cos(lat1) * cos(lat2) * cos(lon1 - lon2);
        ang = ang > 1.0 ? 1.0 : (ang < -1.0 ? -1.0 : ang);
        return acos(ang);
    }
    // euclidean_distance, evaluate_covariance.cpp:28-37 (z = 0 for planar points)
    double dx = b.c0 - a.c0, dy = b.c1 - a.c1, dz = b.c2 - a.c2;
    return sqrt(dx * dx + dy * dy + dz * dz);
}

__device__ __forceinline__ double matern(int nu_x2, double h) {
    if (nu_x2 == 3) {
        double s = 1.7320508075688772 * h;
        return (1.0 + s) * exp(-s);
    }
    return exp(-h);
}

__device__ __forceinline__ float matern_f(int nu_x2, float h) {
    if (nu_x2 == 3) {
        float s = 1.7320508f * h;
        return (1.0f + s) * expf(-s);
    }
    return expf(-h);
}

// C(s1, s2) with per-point sigma^2 (s) and beta (b): evaluate_covariance.cpp:218-225
// (nonstationary) and :82 (stationary: s1 = sill, b1 = range).
// For the straight-line distances the scaled distance over sqrt(bbar^2) is
// taken as sqrt(d^2 / bbar^2) with one reciprocal of bbar^2 shared with the
// prefactor (one division and one square root fewer than the literal form;
// the results agree to a few units in the last place).
__device__ __forceinline__ double cov_entry(const Geom& g, const Pt& p1, double s1, double b1, const Pt& p2,
                                            double s2, double b2) {
    if (g.distance == 1 || !g.nonstat) {
        double D = g.dist_scale * point_distance(g, p1, p2);
        if (!g.nonstat) return s1 * matern(g.nu_x2, D / b1);
        double bms = (b1 * b1 + b2 * b2) / 2;
        double x = (b1 * b2) / bms;
        double pre = g.pref_kind == 0 ? x * sqrt(x) : (g.pref_kind == 1 ? x : pow(x, g.pref_exp));
        return sqrt(s1 * s2) * pre * matern(g.nu_x2, D / sqrt(bms));
    }
    double dx = p2.c0 - p1.c0, dy = p2.c1 - p1.c1, dz = p2.c2 - p1.c2;
    double d2 = dx * dx + dy * dy + dz * dz;
    double ibms = 2.0 / (b1 * b1 + b2 * b2);
    double x = (b1 * b2) * ibms;
    double pre = g.pref_kind == 0 ? x * sqrt(x) : (g.pref_kind == 1 ? x : pow(x, g.pref_exp));
    double h = g.dist_scale * sqrt(d2 * ibms);
    return sqrt(s1 * s2) * pre * matern(g.nu_x2, h);
}

// The same entry evaluated in FP32 (the mixed path's covariance evaluation).
__device__ __forceinline__ float cov_entry_f(const Geom& g, const Pt& p1, float s1, float b1, const Pt& p2, float s2,
                                             float b2) {
    float D;
    if (g.distance == 1) {
        D = (float)(g.dist_scale * point_distance(g, p1, p2));
    } else {
        float dx = (float)(p2.c0 - p1.c0), dy = (float)(p2.c1 - p1.c1), dz = (float)(p2.c2 - p1.c2);
        D = (float)g.dist_scale * sqrtf(dx * dx + dy * dy + dz * dz);
    }
    if (!g.nonstat) return s1 * matern_f(g.nu_x2, D / b1);
    float bms = (b1 * b1 + b2 * b2) * 0.5f;
    float x = (b1 * b2) / bms;
    float pre = g.pref_kind == 0 ? x * sqrtf(x) : (g.pref_kind == 1 ? x : powf(x, (float)g.pref_exp));
    return sqrtf(s1 * s2) * pre * matern_f(g.nu_x2, D / sqrtf(bms));
}

// A point set laid out SoA: coordinates c0/c1/c2 and fields s2 (sigma^2),
// beta, t2 (tau^2), ss (sigma), all indexed by the same global point index.
struct PointSet {
    const double* c0;
    const double* c1;
    const double* c2;
    const double* s2;
    const double* beta;
    const double* t2;
    const double* ss;
    __device__ __forceinline__ Pt pt(long i) const { return Pt{c0[i], c1[i], c2[i]}; }
};


// ----------------------------------------------------------------------------
// tensor-pipe fragments
// ----------------------------------------------------------------------------
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// ----------------------------------------------------------------------------
// CTA-cooperative dense linear algebra (column-major)
// ----------------------------------------------------------------------------
constexpr int TM = 64, TN = 64, TK = 16, NB = 16;

// FP64 products (T = double): CTA tile 64 x (16 NW), NW in {1, 2, 4} picked by
// the width of the product, K slabs of 32.  Each operand tile is staged in
// shared memory in the layout of its global storage -- K-contiguous operands
// as [row][k] (stride 36), the others as [k][row] (stride 68) -- so that the
// coalesced global reads, the staging stores and the m8n8k4 fragment loads
// are all free of bank conflicts (both strides are 4 mod 16 doubles).
constexpr int TK64 = 32;
constexpr int KS64 = TK64 + 4;
constexpr int RS64 = 64 + 4;
constexpr int TILE64 = 64 * KS64;  // >= TK64 * RS64

template <typename T>
struct TilePad;
template <>
struct TilePad<double> {
    static constexpr int v = 4;
};
template <>
struct TilePad<float> {
    static constexpr int v = 8;  // row stride 72 floats: conflict-free m16n8k8 fragment loads
};

template <typename T>
struct LaSmem;
template <>
struct LaSmem<double> {
    double A[2][TILE64];   // two pipeline stages of each operand tile
    double B[2][TILE64];
    double D[NB][NB + 1];  // staged diagonal block
    double inv[NB];        // reciprocals of its diagonal
    double red[kThreads / 32];
    int flag;
};
template <>
struct LaSmem<float> {
    float A[TK][TM + TilePad<float>::v];
    float B[TK][TN + TilePad<float>::v];
    double D[NB][NB + 1];  // staged diagonal block (always FP64)
    double inv[NB];
    double red[kThreads / 32];
    int flag;
};

// The region kernels keep their LaSmem in dynamic shared memory (the FP64
// version is larger than the 48 KB static limit).
template <typename T>
__device__ __forceinline__ LaSmem<T>& la_smem() {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    return *reinterpret_cast<LaSmem<T>*>(la_dyn_smem);
}

// ---- FP64 elementary functions of the covariance entries ----
// The fills are bound by instruction issue and the FP64 pipe, so the entry is
// written for few instructions of both kinds: coefficients come from constant
// memory (a DFMA reads them there; as immediates they cost two moves each), range
// checks and exponents are integer operations on the high word, and one inverse
// square root serves the distance and the prefactor.  Per entry of a 32-lane warp 155 -> 98
// instructions issued; blocks of 1,024 regions of 64 knots with 5 ancestors: 144 ->
// 109 us (230 G entries/s).
static __constant__ double c_exp[15] = {
    1.4426950408889634,      // 1 / ln 2
    6755399441055744.0,      // 1.5 * 2^52: rounds to an integer in the low word
    0.6931471803691238,      // ln 2, 32-bit head (n * head exact)
    1.9082149292705877e-10,  // and tail
    1.6059043836821613e-10, 2.08767569878681e-09, 2.505210838544172e-08, 2.755731922398589e-07,
    2.7557319223985893e-06, 2.48015873015873e-05, 0.0001984126984126984, 0.001388888888888889,
    0.008333333333333333, 0.041666666666666664, 0.16666666666666666};  // 1/13! .. 1/3!

__device__ __forceinline__ unsigned hi_word(double x) { return (unsigned)__double2hiint(x); }

// e^{-s} for s >= 0: Cody-Waite reduction s = n ln2 + r, |r| <= ln2/2; e^{-r} from
// its Taylor polynomial of degree 13 in Horner form (truncation below 5e-18
// relative); 2^{-n} added to the exponent field.  Within 1 ulp of exp(-s) up to
// s = 700; beyond it, and for a negative or undefined s (exp_neg_ok), the result is
// e^{-700}, below 1e-303.
__device__ __forceinline__ bool exp_neg_ok(double s) { return hi_word(s) < 0x4085E000u; }
__device__ __forceinline__ double exp_neg(double s) {
    s = __hiloint2double((int)min(hi_word(s), 0x4085E000u), __double2loint(s));
    const double t = fma(s, c_exp[0], c_exp[1]);
    const double n = t - c_exp[1];
    double u = fma(n, c_exp[2], -s);
    u = fma(n, c_exp[3], u);  // -r
    double p = c_exp[4];
#pragma unroll
    for (int k = 5; k < 15; ++k) p = fma(p, u, c_exp[k]);
    p = fma(p, u, 0.5);
    p = fma(p, u, 1.0);
    p = fma(p, u, 1.0);
    return __hiloint2double(__double2hiint(p) - (__double2loint(t) << 20), __double2loint(p));
}

// 1/sqrt(x): the single-precision approximation (relative error near 2^-23) refined
// by one third-order Householder step y (1 + e/2 + 3 e^2/8), e = 1 - x y^2, which
// takes the error below 2^-66: within an ulp of the exact value.  x must be in
// [2^-100, 2^100) (rsqrt_ok), where the single-precision seed is normal.
__device__ __forceinline__ bool rsqrt_ok(double x) { return hi_word(x) - 0x39B00000u < 0x0C800000u; }
__device__ __forceinline__ double rsqrt_parts(double x, double& c) {  // 1/sqrt(x) = y (1 + c), y of 24 bits
    float yf;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(__double2float_rn(x)));
    const double y = (double)yf;
    const double s = x * y;  // e = 1 - x y^2 with the rounding of x y taken back: the distance enters an exponential
    const double e = fma(-fma(x, y, -s), y, fma(-s, y, 1.0));
    c = e * fma(0.375, e, 0.5);
    return y;
}
__device__ __forceinline__ double rsqrt_seeded(double x) {
    double c;
    const double y = rsqrt_parts(x, c);
    return fma(y, c, y);
}
// a / sqrt(x) from the parts, without rounding 1/sqrt(x) first: lo is the rest that hi + lo rounds
__device__ __forceinline__ double times_parts(double a, double y, double c, double& lo) {
    const double hi = a * y;
    lo = fma(hi, c, fma(a, y, -hi));
    return hi;
}

// One nonstationary straight-line entry from per-point quantities (sqrt(s1 s2)
// pre(x) matern(h), x = 2 b1 b2 / (b1^2 + b2^2), h = scale sqrt(2 d^2 / (b1^2 + b2^2))):
// with g = b^2 / 2 per point and b = g1 + g2, h = scale sqrt(d^2 / b) and x = b1 b2 /
// b.  q = 1/sqrt(d^2 b) gives sqrt(d^2 / b) = d^2 q and 1/b = d^2 q^2, refined by one
// Newton step.  Row point
// (pc, ga, ca = sqrt(s1) b1 for PREF 1; sa = s1, ba for PREF 0), column point (q*, gq,
// ssbq = sqrt(s2) b2; sq = s2, bq).  NU: 1 exponential, 3 Matern 3/2; PREF: 0 prefactor x^1.5, 1 prefactor x;
// SAFE = false sets `bad` where an argument is out of
// rsqrt_seeded's range (coincident points, extreme scales, NaN) and the caller takes
// the SAFE form: tested once per batch of entries, so that the entries' dependent
// chains interleave (a branch in each entry serialised them, 125 us where this form
// takes 109).  Exponents beyond exp_neg's range give e^{-700}, which serves inside an evaluation.
template <int NU, int PREF, bool SAFE>
__device__ __forceinline__ double cov_fast_entry(double pc0, double pc1, double pc2, double ga, double ca,
                                                 double sa, double ba, double qx, double qy, double qz, double gq,
                                                 double ssbq, double sq, double bq, double scale, bool& bad) {
    const double dx = qx - pc0, dy = qy - pc1, dz = qz - pc2;
    const double d2 = fma(dx, dx, fma(dz, dz, dy * dy));
    const double b = ga + gq;
    double h, w;
    if (SAFE) {
        w = 1.0 / b;
        h = sqrt(d2 * w);
    } else {
        const double z = d2 * b;
        bad = bad || !rsqrt_ok(z);
        const double q = rsqrt_seeded(z);
        h = d2 * q;
        w = h * q;
        w = fma(w, fma(-b, w, 1.0), w);
    }
    h *= scale;
    if (NU == 3) h *= 1.7320508075688772;
    const double em = SAFE ? exp(-h) : exp_neg(h);
    const double m = NU == 3 ? fma(h, em, em) : em;
    if (PREF == 1) return (ca * ssbq) * w * m;
    const double x = ba * bq * w, y = sa * sq * x;  // sqrt(s1 s2) x^1.5 = x sqrt(s1 s2 x)
    if (!SAFE) bad = bad || !rsqrt_ok(y);
    const double sy = SAFE ? sqrt(y) : y * rsqrt_seeded(y);
    return x * sy * m;
}

// The same entry where the block is a result by itself, with fewer roundings: the
// exponent is rounded once from d^2 / sqrt(d^2 b) in two parts and the scale (Matern
// 3/2: the scale times sqrt(3), in two parts), c = sqrt(s) b once per point
// (root_times), sqrt(s1 s2 x) once.  An exponent beyond exp_neg's range, negative or
// undefined makes the batch `bad` too.
// Norm of the error against extended precision, fields included, 1500 x 1300 points,
// Matern 1/2 and 3/2, literal form (a division, two square roots, exp) / cov_fast_entry /
// this: chordal 6.67 / 6.72 / 6.67 and 7.16 / 7.20 / 7.11 e-16, planar 3.08 / 3.23 / 3.15
// and 3.41 / 3.52 / 3.40 e-16; against the 64-bit expression 3.08 / 3.18 / 3.10, 3.29 /
// 3.43 / 3.37, 2.39 / 2.43 / 2.26 and 2.60 / 2.63 / 2.52 e-16.  66 us for 4001 x 3003
// planar entries instead of 63, with k_cov_tiles at four CTAs per SM.
struct CovScale {
    double scale, hi, lo;  // distance scale; hi + lo: the exponent's factor, scale or sqrt(3) scale
};
template <int NU, int PREF, bool SAFE>
__device__ __forceinline__ double cov_result_entry(double pc0, double pc1, double pc2, double ga, double ca, double sa,
                                                   double ba, double qx, double qy, double qz, double gq, double cq,
                                                   double sq, double bq, const CovScale& k, bool& bad) {
    const double dx = qx - pc0, dy = qy - pc1, dz = qz - pc2;
    const double d2 = fma(dx, dx, fma(dz, dz, dy * dy));
    const double b = ga + gq;
    double h, w;
    if (SAFE) {
        w = 1.0 / b;
        h = k.scale * sqrt(d2 * w);
        if (NU == 3) h *= 1.7320508075688772;
    } else {
        const double z = d2 * b;
        bad = bad || !rsqrt_ok(z);
        double c, lo;
        const double y = rsqrt_parts(z, c), s = times_parts(d2, y, c, lo);  // sqrt(d^2 / b) = s + lo
        lo *= k.hi;
        if (NU == 3) lo = fma(k.lo, s, lo);
        h = fma(k.hi, s, lo);
        bad = bad || !exp_neg_ok(h);
        w = s * y;  // 1/b to 2^-23, then a third-order step
        const double e = fma(-b, w, 1.0);
        w = fma(w, fma(e, e, e), w);
    }
    const double em = SAFE ? exp(-h) : exp_neg(h);
    const double m = NU == 3 ? fma(h, em, em) : em;
    if (PREF == 1) return (ca * cq) * w * m;
    const double x = ba * bq * w, v = sa * sq * x;
    if (SAFE) return x * sqrt(v) * m;
    bad = bad || !rsqrt_ok(v);
    double c, lo;
    const double y = rsqrt_parts(v, c), r = times_parts(v, y, c, lo);
    return x * (r + lo) * m;
}
// sqrt(|s|) b
__device__ __forceinline__ double root_times(double s, double b) {
    s = fabs(s);
    if (!rsqrt_ok(s)) return sqrt(s) * b;
    double c, lo;
    const double y = rsqrt_parts(s, c), r = times_parts(s, y, c, lo);
    return fma(r, b, lo * b);
}

// One row point against the staged column points q_begin, q_begin + q_step,
// ... < q_end (straight-line distance, nonstationary): writes ob[(qoff + q) ld].
template <typename T, int NU, int PREF>
__device__ __noinline__ void fill_row_fast(const double* __restrict__ sx, const double* __restrict__ sy,
                                           const double* __restrict__ sz, const double* __restrict__ ss,
                                           const double* __restrict__ sb, const double* __restrict__ sg,
                                           const double* __restrict__ ssb, double pc0, double pc1, double pc2,
                                           double sa, double ba, double ga, double scale, int q_begin, int q_end,
                                           int q_step, int qoff, T* __restrict__ ob, long ld) {
    const double ca = sa * ba;  // PREF 1: sa is sqrt(s1)
    for (int q = q_begin; q < q_end; q += 4 * q_step) {
        double v[4];
        bool bad = false;
        auto entry = [&](int k, auto safe) {
            const int e = q + k * q_step < q_end ? q + k * q_step : q;
            v[k] = cov_fast_entry<NU, PREF, decltype(safe)::value>(
                pc0, pc1, pc2, ga, ca, sa, ba, sx[e], sy[e], sz[e], sg[e], PREF == 1 ? ssb[e] : 0.0,
                PREF == 1 ? 0.0 : ss[e], PREF == 1 ? 0.0 : sb[e], scale, bad);
        };
#pragma unroll
        for (int k = 0; k < 4; ++k) entry(k, std::false_type());
        if (bad) {
#pragma unroll
            for (int k = 0; k < 4; ++k) entry(k, std::true_type());
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (q + k * q_step < q_end) ob[(long)(qoff + q + k * q_step) * ld] = (T)v[k];
    }
}

// out[t + q*ld] = C(A_{a0+t}, B_{b0+q}), t < na, q < nb.  When `self` the
// diagonal (t == q) is sigma^2 + tau^2 (evaluate_covariance.cpp:103,307).
// The column points (coordinates, sigma^2 or its root, beta and two products) are staged in
// shared memory in chunks, each thread keeps one row point in registers and
// walks columns strided by the number of row groups (consecutive threads
// write consecutive rows).  The straight-line nonstationary FP64 case with
// the prefactor exponents 1.5 or 1 goes through fill_row_fast; the others
// evaluate cov_entry / cov_entry_f per entry.  Ends with a barrier; uses the
// tile buffers of sm.
// fill_cov_blocks: nblk blocks of na rows each, block k from the row points
// starting at a0[k], written to out + k * blk (same columns for every block);
// `self` applies to block 0 only.
// fill_cov_staged: the same with the staging area given explicitly (7 CH
// doubles) and CH columns staged per chunk; every entry is computed by the same
// per-entry code whatever CH is.
template <typename T, int CH>
__device__ __noinline__ void fill_cov_staged(const Geom& g, const PointSet& P, const long* a0, int nblk, int na,
                                             long b0, int nb, bool self, T* out, long ld, long blk,
                                             double* stage) {
    double* sx = stage;
    double* sy = sx + CH;
    double* sz = sy + CH;
    double* ss = sz + CH;
    double* sb = ss + CH;
    double* sg = sb + CH;   // FP64 fast path only: beta^2 / 2 and sqrt(sigma^2) beta
    double* ssb = sg + CH;  // (7 CH doubles fit the FP64 tile buffers)
    const int tid = threadIdx.x, nt = blockDim.x;
    const int R = nblk * na;  // all rows of all blocks
    const int rows = R < nt ? R : nt;
    const int cols = nt / rows;
    const bool worker = tid < rows * cols;
    const int tr = tid % rows, tq = tid / rows;
    const int nu = g.nu_x2, pk = g.pref_kind;
    const bool fast = sizeof(T) == 8 && fast_form(g);
    const double scale = fabs(g.dist_scale);  // as in cov_block
    for (int q0 = 0; q0 < nb; q0 += CH) {
        const int qn = nb - q0 < CH ? nb - q0 : CH;
        __syncthreads();
        for (int e = tid; e < qn; e += nt) {
            const long ib = b0 + q0 + e;
            sx[e] = P.c0[ib];
            sy[e] = P.c1[ib];
            sz[e] = P.c2[ib];
            ss[e] = fast && pk == 1 ? P.ss[ib] : P.s2[ib];
            const double bb = P.beta[ib];
            sb[e] = bb;
            if (fast) {
                sg[e] = 0.5 * (bb * bb);
                ssb[e] = ss[e] * bb;
            }
        }
        __syncthreads();
        if (!worker) continue;
        for (int tt = tr; tt < R; tt += rows) {
            const int kb = tt / na, t = tt - kb * na;
            const long ia = a0[kb] + t;
            if (fast) {
                T* ob = out + kb * blk + t;
                const double pc0 = P.c0[ia], pc1 = P.c1[ia], pc2 = P.c2[ia];
                const double sa = P.s2[ia], ba = P.beta[ia];
                const double ssa = pk == 1 ? P.ss[ia] : sa, ga = 0.5 * (ba * ba);
                if (nu == 3 && pk == 1)
                    fill_row_fast<T, 3, 1>(sx, sy, sz, ss, sb, sg, ssb, pc0, pc1, pc2, ssa, ba, ga, scale, tq, qn, cols,
                                           q0, ob, ld);
                else if (nu == 3)
                    fill_row_fast<T, 3, 0>(sx, sy, sz, ss, sb, sg, ssb, pc0, pc1, pc2, ssa, ba, ga, scale, tq, qn, cols,
                                           q0, ob, ld);
                else if (pk == 1)
                    fill_row_fast<T, 1, 1>(sx, sy, sz, ss, sb, sg, ssb, pc0, pc1, pc2, ssa, ba, ga, scale, tq, qn, cols,
                                           q0, ob, ld);
                else
                    fill_row_fast<T, 1, 0>(sx, sy, sz, ss, sb, sg, ssb, pc0, pc1, pc2, ssa, ba, ga, scale, tq, qn, cols,
                                           q0, ob, ld);
                // the diagonal of a self block, whose entry this thread has just written
                if (self && kb == 0) {
                    const int qd = t - q0;
                    if (qd >= tq && qd < qn && (qd - tq) % cols == 0) ob[(long)t * ld] = (T)(sa + P.t2[ia]);
                }
                continue;
            }
            T* ob = out + kb * blk;
            const Pt pa = P.pt(ia);
            const double sa = P.s2[ia], ba = P.beta[ia];
#pragma unroll 4
            for (int q = tq; q < qn; q += cols) {
                const int qq = q0 + q;
                T v;
                if (self && kb == 0 && t == qq) {
                    v = (T)(sa + P.t2[ia]);
                } else if (sizeof(T) == 8) {
                    v = (T)cov_entry(g, pa, sa, ba, Pt{sx[q], sy[q], sz[q]}, ss[q], sb[q]);
                } else {
                    v = (T)cov_entry_f(g, pa, (float)sa, (float)ba, Pt{sx[q], sy[q], sz[q]}, (float)ss[q],
                                       (float)sb[q]);
                }
                ob[t + (long)qq * ld] = v;
            }
        }
    }
    __syncthreads();
}

template <typename T>
__device__ inline void fill_cov_blocks(const Geom& g, const PointSet& P, const long* a0, int nblk, int na, long b0,
                                       int nb, bool self, T* out, long ld, long blk, LaSmem<T>& sm) {
    // the staging area is the tile buffers of sm: 7 CH doubles
    fill_cov_staged<T, sizeof(T) == 8 ? 512 : 96>(g, P, a0, nblk, na, b0, nb, self, out, ld, blk,
                                                   reinterpret_cast<double*>(&sm.A[0][0]));
}

template <typename T>
__device__ inline void fill_cov(const Geom& g, const PointSet& P, long a0, int na, long b0, int nb, bool self,
                                T* out, long ld, LaSmem<T>& sm) {
    fill_cov_blocks<T>(g, P, &a0, 1, na, b0, nb, self, out, ld, 0, sm);
}

constexpr int kCovThreads = 256;
constexpr int kCovChunk = 64;  // column points staged per chunk (7 x 64 doubles of shared memory, 16-byte aligned)

// The straight-line nonstationary FP64 block: two row points per thread with their
// parameters in registers, the column points staged in chunks as pairs (x, y), (z,
// g), (sqrt(s2) b or s2, b), which both rows read.
// self: row t is the point of column t + doff.
// RESULT: the entries are a result by themselves (cov_result_entry).
template <typename T, int NU, int PREF, bool RESULT = false>
__device__ __forceinline__ void cov_block_fast(const PointSet& P, long a0, int nr, long b0, int nc, bool self, int doff,
                                               T* __restrict__ out, long ld, const CovScale& scale, double* stage) {
    double2* sxy = reinterpret_cast<double2*>(stage);
    double2* szg = sxy + kCovChunk;
    double2* s45 = szg + kCovChunk;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int half = (nr + 1) / 2;
    const int rows = half < nt ? half : nt;
    const int cols = nt / rows;
    const bool worker = tid < rows * cols;
    const int tr = tid % rows, tc = tid / rows;
    for (int q0 = 0; q0 < nc; q0 += kCovChunk) {
        const int qn = nc - q0 < kCovChunk ? nc - q0 : kCovChunk;
        __syncthreads();
        for (int e = tid; e < qn; e += nt) {
            const long ib = b0 + q0 + e;
            const double bb = P.beta[ib], sq = PREF == 1 && !RESULT ? P.ss[ib] : P.s2[ib];
            sxy[e] = make_double2(P.c0[ib], P.c1[ib]);
            szg[e] = make_double2(P.c2[ib], 0.5 * (bb * bb));
            s45[e] = make_double2(PREF == 1 ? (RESULT ? root_times(sq, bb) : sq * bb) : sq, bb);
        }
        __syncthreads();
        if (!worker) continue;
        for (int t = tr; t < half; t += rows) {
            const bool two = t + half < nr;
            double pc0[2], pc1[2], pc2[2], ga[2], ca[2], sa[2], bt[2], diag[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const long ia = a0 + t + (k && two ? half : 0);
                const double ba = P.beta[ia];
                pc0[k] = P.c0[ia];
                pc1[k] = P.c1[ia];
                pc2[k] = P.c2[ia];
                sa[k] = PREF == 1 && !RESULT ? P.ss[ia] : P.s2[ia];
                ga[k] = 0.5 * (ba * ba);
                bt[k] = ba;
                ca[k] = PREF == 1 && RESULT ? root_times(sa[k], ba) : sa[k] * ba;
                diag[k] = self ? P.s2[ia] + P.t2[ia] : 0.0;
            }
            T* ob = out + t + (long)(q0 + tc) * ld;
            const long step = (long)cols * ld;
            for (int q = tc; q < qn; q += 2 * cols, ob += 2 * step) {
                const int qb = q + cols < qn ? q + cols : q;  // two columns at a time: four entries
                double v[4];
                bool bad = false;
                auto entry = [&](int e, auto safe) {
                    const int k = e & 1, c = e < 2 ? q : qb;
                    const double2 xy = sxy[c], zg = szg[c], r45 = s45[c];
                    bool b1 = false;
                    if constexpr (RESULT)
                        v[e] = cov_result_entry<NU, PREF, decltype(safe)::value>(
                            pc0[k], pc1[k], pc2[k], ga[k], ca[k], sa[k], bt[k], xy.x, xy.y, zg.x, zg.y, r45.x, r45.x,
                            r45.y, scale, b1);
                    else
                        v[e] = cov_fast_entry<NU, PREF, decltype(safe)::value>(
                            pc0[k], pc1[k], pc2[k], ga[k], ca[k], sa[k], bt[k], xy.x, xy.y, zg.x, zg.y, r45.x, r45.x,
                            r45.y, scale.scale, b1);
                    bad = bad || (b1 && !(self && t + k * half + doff == q0 + c));  // the diagonal is replaced below
                };
#pragma unroll
                for (int e = 0; e < 4; ++e) entry(e, std::false_type());
                if (bad) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) entry(e, std::true_type());
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int k = e & 1, c = e < 2 ? q : qb;
                    if (self && t + k * half + doff == q0 + c) v[e] = diag[k];  // sigma^2 + tau^2 (evaluate_covariance.cpp:103,307)
                    if ((k == 0 || two) && (e < 2 || q + cols < qn)) ob[k * half + (e < 2 ? 0 : step)] = (T)v[e];
                }
            }
        }
    }
    __syncthreads();
}

template <int KIND>
struct CovForm {
    static constexpr int NU = KIND < 3 ? 3 : 1, PREF = KIND & 1;
};

// Block out[t + q ld] = C(A_{a0+t}, B_{b0+q}), t < nr, q < nc (with the
// sigma^2 + tau^2 diagonal when `self`), by the whole CTA.  KIND (cov_kind on the
// host): 1..4 the straight-line nonstationary FP64 forms (Matern 3/2 or 1/2 x
// prefactor exponent 1 or 3/2), 0 every other model.  Planar points take them with all
// three coordinates, as every other kernel does (without the third, which their readers
// write as zero, an entry takes two instructions less: 60 us instead of 63 for 4001 x 3003).
// CH: column points staged per chunk by the other models (7 CH doubles of stage).
template <typename T, int KIND, int CH = kCovChunk>
__device__ __forceinline__ void cov_block(const Geom& g, const PointSet& P, long a0, int nr, long b0, int nc, bool self,
                                          T* out, long ld, double* stage) {
    if constexpr (KIND == 0) {
        fill_cov_staged<T, CH>(g, P, &a0, 1, nr, b0, nc, self, out, ld, 0, stage);
    } else {
        using F = CovForm<KIND>;
        // an evaluation's straight-line distances take the scale's magnitude
        cov_block_fast<T, F::NU, F::PREF>(P, a0, nr, b0, nc, self, 0, out, ld, CovScale{fabs(g.dist_scale), 0.0, 0.0},
                                          stage);
    }
}

inline int cov_kind(const Geom& g, bool fp64) {
    if (!fp64 || !fast_form(g)) return 0;
    return g.nu_x2 == 3 ? (g.pref_kind == 1 ? 1 : 2) : (g.pref_kind == 1 ? 3 : 4);
}

// Calls f(std::integral_constant<int, KIND>) for the model's form.
template <typename Fn>
inline void with_cov_kind(int kind, Fn&& f) {
    switch (kind) {
        case 1: f(std::integral_constant<int, 1>()); break;
        case 2: f(std::integral_constant<int, 2>()); break;
        case 3: f(std::integral_constant<int, 3>()); break;
        case 4: f(std::integral_constant<int, 4>()); break;
        default: f(std::integral_constant<int, 0>()); break;
    }
}


// ---- FP64: warp tile (8 NW) rows x 16 columns --------------------------------
template <int NW>
struct AccD {
    double v[NW][2][2];  // NW (m8) x 2 (n8) fragments of m8n8
};

// 8-byte asynchronous global -> shared copy; pred == false writes zeros.
__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool pred) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = pred ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}
// 16-byte asynchronous global -> shared copy through L2 only; pred == false
// writes zeros (src must then still be a valid 16-byte aligned address).
__device__ __forceinline__ void cp_async16z(double* dst, const double* src, bool pred) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = pred ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}
// Bulk prefetch into L2 of the 16-byte aligned part of [p, p + bytes) (the
// instruction takes a 16-byte aligned address and a multiple of 16 bytes).
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned long bytes) {
    const unsigned long a = ((unsigned long)p + 15) & ~15ul, b = ((unsigned long)p + bytes) & ~15ul;
    if (b <= a || b - a > 0xffffffffull) return;
    asm volatile(
        "{\n\t.reg .u64 ga;\n\tcvta.to.global.u64 ga, %0;\n\tcp.async.bulk.prefetch.L2.global [ga], %1;\n\t}\n" ::"l"(a),
        "r"((unsigned)(b - a))
        : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <bool TA, bool TB, int NW>
__device__ __forceinline__ void warp_step_f64(AccD<NW>& acc, const double* sA, const double* sB, int wm, int wn,
                                              int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int k4 = 0; k4 < TK64; k4 += 4) {
        double a[NW], b[2];
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            const int row = wm + 8 * i + g, k = k4 + t;
            a[i] = TA ? sA[row * KS64 + k] : sA[k * RS64 + row];
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int col = wn + 8 * j + g, k = k4 + t;
            b[j] = TB ? sB[k * RS64 + col] : sB[col * KS64 + k];
        }
#pragma unroll
        for (int i = 0; i < NW; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) mma_f64(acc.v[i][j], a[i], b[j]);
    }
}

// Operands must be in global memory (they are copied with cp.async): a
// two-stage pipeline keeps the next K slab in flight while the tensor pipe
// works on the current one.
template <bool TA, bool TB, int NW>
__device__ inline void gemm_f64(int M, int N, int K, double alpha, const double* A, long lda, const double* B,
                                long ldb, double beta, double* C, long ldc, LaSmem<double>& sm,
                                const double* Cin = nullptr, long ldcin = 0) {
    constexpr int W = 16 * NW;                // CTA tile width
    constexpr int WM = 8 / NW;                // warps along M
    constexpr int PA = 64 * TK64 / kThreads;  // A elements per thread per slab (8)
    constexpr int PB = W * TK64 / kThreads;   // B elements per thread per slab (2 NW)
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int wm = (w % WM) * 8 * NW, wn = (w / WM) * 16;
    for (int m0 = 0; m0 < M; m0 += 64) {
        for (int n0 = 0; n0 < N; n0 += W) {
            AccD<NW> acc;
#pragma unroll
            for (int i = 0; i < NW; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) acc.v[i][j][0] = acc.v[i][j][1] = 0.0;
            auto issue = [&](int k0, int stage) {
                double* sA = sm.A[stage];
                double* sB = sm.B[stage];
#pragma unroll
                for (int q = 0; q < PA; ++q) {
                    const int e = tid + q * kThreads;
                    // TA: op(A)[i][k] = A[k + i lda] (K-contiguous), else A[i + k lda]
                    const int i = TA ? e / TK64 : e % 64, k = TA ? e % TK64 : e / 64;
                    const int gi = m0 + i, gk = k0 + k;
                    const bool ok = gi < M && gk < K;
                    const double* src = ok ? (TA ? A + gk + (long)gi * lda : A + gi + (long)gk * lda) : A;
                    cp_async8(sA + (TA ? i * KS64 + k : k * RS64 + i), src, ok);
                }
#pragma unroll
                for (int q = 0; q < PB; ++q) {
                    const int e = tid + q * kThreads;
                    // TB: op(B)[k][j] = B[j + k ldb], else B[k + j ldb] (K-contiguous)
                    const int j = TB ? e % W : e / TK64, k = TB ? e / W : e % TK64;
                    const int gj = n0 + j, gk = k0 + k;
                    const bool ok = gj < N && gk < K;
                    const double* src = ok ? (TB ? B + gj + (long)gk * ldb : B + gk + (long)gj * ldb) : B;
                    cp_async8(sB + (TB ? k * RS64 + j : j * KS64 + k), src, ok);
                }
                cp_async_commit();
            };
            // warps whose tile lies outside the product skip the tensor work
            const bool active = m0 + wm < M && n0 + wn < N;
            if (K > 0) issue(0, 0);
            int stage = 0;
            for (int k0 = 0; k0 < K; k0 += TK64, stage ^= 1) {
                if (k0 + TK64 < K) {
                    issue(k0 + TK64, stage ^ 1);
                    cp_async_wait<1>();
                } else {
                    cp_async_wait<0>();
                }
                __syncthreads();
                if (active) warp_step_f64<TA, TB, NW>(acc, sm.A[stage], sm.B[stage], wm, wn, lane);
                __syncthreads();
            }
            if (active) {
                const int g = lane >> 2, t = lane & 3;
#pragma unroll
                for (int i = 0; i < NW; ++i)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int r = m0 + wm + 8 * i + g, c = n0 + wn + 8 * j + 2 * t;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if (r < M && c + h < N) {
                                double* p = C + r + (long)(c + h) * ldc;
                                const double* q = Cin ? Cin + r + (long)(c + h) * ldcin : p;
                                *p = beta == 0.0 ? alpha * acc.v[i][j][h] : alpha * acc.v[i][j][h] + beta * *q;
                            }
                        }
                    }
            }
        }
    }
    __syncthreads();
}

// ---- FP32 storage (mixed path): 3xTF32 products, 64 x 64 tiles, K slabs of 16
struct AccF {
    float v[2][2][4];  // 2 (m16) x 2 (n8) fragments of m16n8
};

__device__ __forceinline__ void warp_step_tf32x3(AccF& acc, const LaSmem<float>& sm, int wm, int wn, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int k8 = 0; k8 < TK; k8 += 8) {
        uint32_t ah[2][4], al[2][4], bh[2][2], bl[2][2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r0 = wm + 16 * i + g;
            float x[4] = {sm.A[k8 + t][r0], sm.A[k8 + t][r0 + 8], sm.A[k8 + t + 4][r0], sm.A[k8 + t + 4][r0 + 8]};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                ah[i][q] = to_tf32(x[q]);
                al[i][q] = to_tf32(x[q] - __uint_as_float(ah[i][q]));
            }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int c0 = wn + 8 * j + g;
            float y[2] = {sm.B[k8 + t][c0], sm.B[k8 + t + 4][c0]};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                bh[j][q] = to_tf32(y[q]);
                bl[j][q] = to_tf32(y[q] - __uint_as_float(bh[j][q]));
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                mma_tf32(acc.v[i][j], al[i], bh[j]);
                mma_tf32(acc.v[i][j], ah[i], bl[j]);
                mma_tf32(acc.v[i][j], ah[i], bh[j]);
            }
    }
}

template <bool TA, bool TB>
__device__ inline void gemm_f32(int M, int N, int K, float alpha, const float* A, long lda, const float* B, long ldb,
                                float beta, float* C, long ldc, LaSmem<float>& sm, const float* Cin = nullptr,
                                long ldcin = 0) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int wm = (w & 1) * 32, wn = (w >> 1) * 16;
    constexpr int PER = TK * TM / kThreads;  // elements of each operand per thread per slab (4)
    for (int m0 = 0; m0 < M; m0 += TM) {
        for (int n0 = 0; n0 < N; n0 += TN) {
            AccF acc;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int q = 0; q < 4; ++q) acc.v[i][j][q] = 0.f;
            float ra[PER], rb[PER];
            auto fetch = [&](int k0) {
#pragma unroll
                for (int q = 0; q < PER; ++q) {
                    const int e = tid + q * kThreads;
                    int i, k;
                    if (!TA) { i = e % TM; k = e / TM; } else { k = e % TK; i = e / TK; }
                    const int gi = m0 + i, gk = k0 + k;
                    ra[q] = (gi < M && gk < K) ? (TA ? A[gk + (long)gi * lda] : A[gi + (long)gk * lda]) : 0.f;
                    int j, kb;
                    if (!TB) { kb = e % TK; j = e / TK; } else { j = e % TN; kb = e / TN; }
                    const int gj = n0 + j, gkb = k0 + kb;
                    rb[q] = (gj < N && gkb < K) ? (TB ? B[gj + (long)gkb * ldb] : B[gkb + (long)gj * ldb]) : 0.f;
                }
            };
            auto stash = [&]() {
#pragma unroll
                for (int q = 0; q < PER; ++q) {
                    const int e = tid + q * kThreads;
                    int i, k;
                    if (!TA) { i = e % TM; k = e / TM; } else { k = e % TK; i = e / TK; }
                    sm.A[k][i] = ra[q];
                    int j, kb;
                    if (!TB) { kb = e % TK; j = e / TK; } else { j = e % TN; kb = e / TN; }
                    sm.B[kb][j] = rb[q];
                }
            };
            if (K > 0) {
                fetch(0);
                stash();
            }
            __syncthreads();
            for (int k0 = 0; k0 < K; k0 += TK) {
                const bool more = k0 + TK < K;
                if (more) fetch(k0 + TK);
                warp_step_tf32x3(acc, sm, wm, wn, lane);
                __syncthreads();
                if (more) {
                    stash();
                    __syncthreads();
                }
            }
            const int g = lane >> 2, t = lane & 3;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int r = m0 + wm + 16 * i + g, c = n0 + wn + 8 * j + 2 * t;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int rr = r + (q >> 1) * 8, cc = c + (q & 1);
                        if (rr < M && cc < N) {
                            float* p = C + rr + (long)cc * ldc;
                            const float* qi = Cin ? Cin + rr + (long)cc * ldcin : p;
                            *p = beta == 0.f ? alpha * acc.v[i][j][q] : alpha * acc.v[i][j][q] + beta * *qi;
                        }
                    }
                }
        }
    }
    __syncthreads();
}

// C = alpha * op(A) * op(B) + beta * Cin (Cin = C unless given, ld ldcin);
// op(A): M x K, op(B): K x N, column-major,
// any leading dimensions; A and B in global memory.  beta == 0 never reads C.
// Ends with a barrier.
// FP64 tile width (NW) per product-width bucket (N <= 16, N <= 32, wider),
// chosen per device by the autotuner (mra_autotune); {1, 2, 4} by default.  Every
// file that includes this holds its own copy (set_gemm_tiles sets them all).
// The choice changes only how output tiles are spread over warps: every
// element is accumulated by one thread in the same K order, so results are
// bitwise the same whatever the choice.
__constant__ int c_gemm_nw[3] = {1, 2, 4};

// ONE_TILE: the product must be computed as one column tile (N <= 64) --
// required when C aliases A (an in-place product C = C X): each row tile then
// reads all of its rows before writing them, whereas a second column tile
// would read columns the first one has already overwritten.
template <typename T, bool TA, bool TB, bool ONE_TILE = false>
__device__ inline void gemm(int M, int N, int K, T alpha, const T* A, long lda, const T* B, long ldb, T beta, T* C,
                            long ldc, LaSmem<T>& sm, const T* Cin = nullptr, long ldcin = 0) {
    if constexpr (sizeof(T) == 8) {
        const int nw = ONE_TILE ? (N <= 16 ? 1 : (N <= 32 ? 2 : 4)) : c_gemm_nw[N <= 16 ? 0 : (N <= 32 ? 1 : 2)];
        if (nw == 1) gemm_f64<TA, TB, 1>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, sm, Cin, ldcin);
        else if (nw == 2) gemm_f64<TA, TB, 2>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, sm, Cin, ldcin);
        else gemm_f64<TA, TB, 4>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, sm, Cin, ldcin);
    } else {
        gemm_f32<TA, TB>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, sm, Cin, ldcin);
    }
}

// Stages the nb x nb diagonal block of L at b0 in FP64 with the reciprocals of
// its diagonal.  Ends with a barrier.
template <typename T>
__device__ inline void stage_diag_block(const T* L, long ldl, int b0, int nb, LaSmem<T>& sm) {
    for (int e = threadIdx.x; e < nb * nb; e += kThreads) {
        int i = e % nb, j = e / nb;
        sm.D[i][j] = (double)L[(b0 + i) + (long)(b0 + j) * ldl];
    }
    __syncthreads();
    if (threadIdx.x < nb) sm.inv[threadIdx.x] = 1.0 / sm.D[threadIdx.x][threadIdx.x];
    __syncthreads();
}

// B <- L^{-1} B  (L: n x n lower, non-unit; B: n x nrhs).  dtrtrs('L','N','N').
// Diagonal blocks are solved in FP64; trailing updates go through gemm<T>.
template <typename T>
__device__ inline void trsm_left_lower(int n, int nrhs, const T* L, long ldl, T* B, long ldb, LaSmem<T>& sm) {
    const int tid = threadIdx.x;
    for (int b0 = 0; b0 < n; b0 += NB) {
        int nb = min(NB, n - b0);
        stage_diag_block(L, ldl, b0, nb, sm);
        for (int c = tid; c < nrhs; c += kThreads) {
            double x[NB];
            T* col = B + b0 + (long)c * ldb;
#pragma unroll
            for (int i = 0; i < NB; ++i) x[i] = i < nb ? (double)col[i] : 0.0;
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
                if (i < nb) col[i] = (T)x[i];
        }
        __syncthreads();
        if (b0 + nb < n)
            gemm<T, false, false>(n - b0 - nb, nrhs, nb, (T)-1, L + (b0 + nb) + (long)b0 * ldl, ldl, B + b0, ldb,
                                  (T)1, B + b0 + nb, ldb, sm);
    }
}

// B <- B L^{-T}  (L: n x n lower; B: rows x n).  Row-wise forward substitution.
template <typename T>
__device__ inline void trsm_right_lower_trans(int rows, int n, const T* L, long ldl, T* B, long ldb, LaSmem<T>& sm) {
    const int tid = threadIdx.x;
    for (int b0 = 0; b0 < n; b0 += NB) {
        int nb = min(NB, n - b0);
        stage_diag_block(L, ldl, b0, nb, sm);
        for (int row = tid; row < rows; row += kThreads) {
            double x[NB];
            T* p = B + row + (long)b0 * ldb;
#pragma unroll
            for (int i = 0; i < NB; ++i) x[i] = i < nb ? (double)p[(long)i * ldb] : 0.0;
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
                if (i < nb) p[(long)i * ldb] = (T)x[i];
        }
        __syncthreads();
        if (b0 + nb < n)
            gemm<T, false, true>(rows, n - b0 - nb, nb, (T)-1, B + (long)b0 * ldb, ldb, L + (b0 + nb) + (long)b0 * ldl,
                                 ldl, (T)1, B + (long)(b0 + nb) * ldb, ldb, sm);
    }
}

// Solves L x = b for one right-hand side entirely in FP64 (the vectors that feed
// quadratic forms), x overwrites b.  Single warp does the work; ends with a barrier.
template <typename T>
__device__ inline void trsv_lower_f64(int n, const T* L, long ldl, double* b) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        for (int i = 0; i < n; ++i) {
            double s = 0.0;
            for (int k = lane; k < i; k += 32) s += (double)L[i + (long)k * ldl] * b[k];
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (lane == 0) b[i] = (b[i] - s) / (double)L[i + (long)i * ldl];
            __syncwarp();
        }
    }
    __syncthreads();
}

// x = Linv b for a lower-triangular Linv (n x n, ld ldl) that is the inverse
// of a factor, stored with exact zeros above its diagonal: the triangular
// solve as a product, one row per thread, every row over all n columns (a
// uniform trip count, unrolled, so the loads of a row are in flight
// together).  x may alias b.  Ends with a barrier.
template <typename T>
__device__ inline void trmv_lower_inv(int n, const T* Linv, long ldl, double* x, const double* b) {
    double v[2] = {0.0, 0.0};
    for (int h = 0; h < 2; ++h) {
        const int q = threadIdx.x + h * kThreads;
        if (q < n) {
            double s[4] = {0.0, 0.0, 0.0, 0.0};
            int k = 0;
            for (; k + 8 <= n; k += 8) {
#pragma unroll
                for (int u = 0; u < 8; ++u) s[u & 3] += (double)Linv[q + (long)(k + u) * ldl] * b[k + u];
            }
            for (; k < n; ++k) s[0] += (double)Linv[q + (long)k * ldl] * b[k];
            v[h] = (s[0] + s[1]) + (s[2] + s[3]);
        }
    }
    __syncthreads();
    for (int h = 0; h < 2; ++h) {
        const int q = threadIdx.x + h * kThreads;
        if (q < n) x[q] = v[h];
    }
    __syncthreads();
}

// Deterministic CTA sum (fixed thread -> element mapping and tree order).
template <typename T>
__device__ inline double cta_sum(double v, LaSmem<T>& sm) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sm.red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kThreads / 32; ++w) s += sm.red[w];
    __syncthreads();
    return s;  // valid in thread 0
}

// In-place lower Cholesky A = L L^T (strict upper part zeroed, like
// Armadillo's chol(X, "lower")).  Diagonal blocks and panels in FP64, trailing
// updates through gemm<T>.  Returns 0, or the 1-based index of the first
// non-positive (or NaN) pivot (LAPACK's info); the factorization then goes on
// with NaNs and the caller reports the region.  *logdet (thread 0) receives
// 2 * sum(log(diag L)) accumulated in FP64.
template <typename T>
__device__ inline int potrf_blocked(int n, T* A, long lda, LaSmem<T>& sm, double* logdet) {
    const int tid = threadIdx.x;
    double ld = 0.0;
    if (tid == 0) sm.flag = 0;
    for (int b0 = 0; b0 < n; b0 += NB) {
        int nb = min(NB, n - b0);
        for (int e = tid; e < nb * nb; e += kThreads) {
            int i = e % nb, j = e / nb;
            sm.D[i][j] = (double)A[(b0 + i) + (long)(b0 + j) * lda];
        }
        __syncthreads();
        // the diagonal block by warp 0, lane i owning row i (right-looking)
        if (tid < 32) {
            const int lane = tid;
            for (int k = 0; k < nb; ++k) {
                if (lane == 0) {
                    double d = sm.D[k][k];
                    if (!(d > 0.0) && sm.flag == 0) sm.flag = b0 + k + 1;
                    double sq = sqrt(d);
                    sm.D[k][k] = sq;
                    sm.inv[k] = 1.0 / sq;
                    ld += 2.0 * log(sq);
                }
                __syncwarp();
                if (lane > k && lane < nb) sm.D[lane][k] *= sm.inv[k];
                __syncwarp();
                // lane i reads column k (final) and writes row i beyond column k
                if (lane > k && lane < nb) {
                    const double lik = sm.D[lane][k];
                    for (int j = k + 1; j <= lane; ++j) sm.D[lane][j] -= lik * sm.D[j][k];
                }
                __syncwarp();
            }
        }
        __syncthreads();
        for (int e = tid; e < nb * nb; e += kThreads) {
            int i = e % nb, j = e / nb;
            A[(b0 + i) + (long)(b0 + j) * lda] = j <= i ? (T)sm.D[i][j] : (T)0;
        }
        __syncthreads();
        int rest = n - b0 - nb;
        if (rest > 0) {
            // panel: A[b0+nb:, b0:b0+nb] <- A[...] * D^{-T}, in FP64
            for (int row = tid; row < rest; row += kThreads) {
                double x[NB];
                T* p = A + (b0 + nb + row) + (long)b0 * lda;
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
                    if (i < nb) p[(long)i * lda] = (T)x[i];
            }
            __syncthreads();
            const T* P = A + (b0 + nb) + (long)b0 * lda;
            gemm<T, false, true>(rest, rest, nb, (T)-1, P, lda, P, lda, (T)1, A + (b0 + nb) + (long)(b0 + nb) * lda,
                                 lda, sm);
            for (int e = tid; e < nb * rest; e += kThreads) {
                int i = e % nb, j = e / nb;
                A[(b0 + i) + (long)(b0 + nb + j) * lda] = (T)0;
            }
            __syncthreads();
        }
    }
    __syncthreads();
    if (tid == 0 && logdet) *logdet = ld;
    return sm.flag;
}


// FP64 Cholesky (and optionally the inverse of the factor) of an n x n
// matrix, n <= 64, staged whole in shared memory (column-major, ld 68: 4 mod 16
// doubles, conflict-free m8n8k4 fragments), right-looking in 8-wide blocks.
// What bounds it is the chain of the 64 pivots (1/sqrt, scale, update), so each
// block's 8 x 8 diagonal is factored redundantly in the registers of every
// thread that needs it -- no shuffles or barriers inside the chain -- and the
// inverse rides along: with X = I to start with, block row k of X = L^{-1} is the
// same 8-step substitution as a panel row, and its update another tile of the
// trailing product.
//  * threads 0..63: row of the panel (the diagonal block's rows among them);
//    threads 64..127: column of X's block row;
//  * all warps: 8 x 8 tiles of the trailing matrix and of X by m8n8k4.
// n that is not a multiple of 8 is padded with an identity block.  A
// non-positive or NaN pivot sets sm.flag (1-based index, first wins) and the
// factorization goes on with NaNs.  logdet (thread 0) = 2 sum log L_ii.
// n = 64 with the inverse, one CTA of 256: 21,100 cycles, n = 16: 5,900 (16-wide
// blocks with the diagonal block's rows in lanes and shuffled pivots: 55,800 and
// 11,800); two CTAs per SM: 27,000 each (62,100).
constexpr int SLD = 68;

// S (N x N valid lower part, N = n rounded up to 8) -> L; X -> L^{-1} if kInv.
// Starts after a barrier on S, ends with one.
// NT (128 or 256): threads of the CTA; LD: row stride of S and X (4 mod 16 doubles).
template <bool kInv, typename Sm, int NT = kThreads, int LD = SLD>
__device__ __forceinline__ void potrf_core(int n, double* S, double* X, Sm& sm) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int nbk = (n + 7) >> 3, N = nbk << 3;
    if (kInv) {
        for (int c = w; c < N; c += NT / 32)
            for (int i = lane; i < N; i += 32) X[i + c * LD] = i == c ? 1.0 : 0.0;
        __syncthreads();
    }
    int bad = 0;
    for (int k = 0; k < nbk; ++k) {
        const int k0 = k << 3;
        const int row = k0 + tid, c = tid - 64;
        const bool prow = tid < 64 && row < N, pcol = kInv && tid >= 64 && c < k0 + 8;
        double* base = tid < 64 ? S + row + k0 * LD : X + k0 + c * LD;
        const int step = tid < 64 ? LD : 1;
        double l[36], x[8];  // the diagonal block, row by row; this thread's panel row or column of X
        if (tid < 128) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) l[i * (i + 1) / 2 + j] = S[(k0 + i) + (k0 + j) * LD];
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = prow || pcol ? base[j * step] : 0.0;
        }
        __syncthreads();  // the block is read before its rows are rewritten
        if (tid < 128) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const double d = l[j * (j + 1) / 2 + j];
                if (!(d > 0.0) && bad == 0 && k0 + j < n) bad = k0 + j + 1;
                const double r = rsqrt(d);
#pragma unroll
                for (int i = j + 1; i < 8; ++i) l[i * (i + 1) / 2 + j] *= r;
                x[j] *= r;
#pragma unroll
                for (int i = j + 1; i < 8; ++i) {
#pragma unroll
                    for (int q = j + 1; q <= i; ++q)
                        l[i * (i + 1) / 2 + q] = fma(-l[i * (i + 1) / 2 + j], l[q * (q + 1) / 2 + j], l[i * (i + 1) / 2 + q]);
                    x[i] = fma(-l[i * (i + 1) / 2 + j], x[j], x[i]);
                }
            }
            if (prow || pcol) {
#pragma unroll
                for (int j = 0; j < 8; ++j) base[j * step] = tid < 64 && j > tid ? 0.0 : x[j];  // zeros above the diagonal
            }
        }
        __syncthreads();
        // trailing tiles by block columns: column q <= k of X (rows below k), column q > k of S (rows from q)
        for (int q = w; q < nbk; q += NT / 32) {
            if (!kInv && q <= k) continue;
            const bool inX = q <= k;
            const double* B = inX ? X + k0 + 8 * q * LD : S + 8 * q + k0 * LD;
            const int bs = inX ? LD : 1, bt = inX ? 1 : LD;
            const double b0 = B[g * bs + t * bt], b1 = B[g * bs + (4 + t) * bt];
            double* C = (inX ? X : S) + g + (8 * q + 2 * t) * LD;
            const double* A = S + g + (k0 + t) * LD;
            int bi = inX ? k + 1 : q;
#pragma unroll 4
            for (; bi < nbk; ++bi) {
                double acc[2] = {-C[8 * bi], -C[8 * bi + LD]};
                mma_f64(acc, A[8 * bi], b0);
                mma_f64(acc, A[8 * bi + 4 * LD], b1);
                C[8 * bi] = -acc[0];
                C[8 * bi + LD] = -acc[1];
            }
        }
        __syncthreads();
    }
    if (tid == 0) sm.flag = bad;
}

// Factors S = sm.A (after a barrier) and writes L to A and, if kInv, its inverse
// (formed in sm.B) to inv, zeros above the diagonals; returns the first bad pivot.
// A function of its own, with its registers to itself; sm is the kernel's dynamic
// shared memory, taken here so that its accesses are known to be shared ones.
template <bool kInv, typename Sm, int NT = kThreads>
__device__ __noinline__ int potrf_finish(int n, double* A, long lda, double* logdet, double* inv, long ldinv) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    Sm& sm = *reinterpret_cast<Sm*>(la_dyn_smem);
    double* S = &sm.A[0][0];
    double* X = &sm.B[0][0];
    const int tid = threadIdx.x;
    potrf_core<kInv, Sm, NT>(n, S, X, sm);
    if (tid < 64) {
        double part = tid < n ? log(S[tid + tid * SLD]) : 0.0;
        for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
        if ((tid & 31) == 0) sm.red[tid >> 5] = part;
    }
    const int i = tid & 63;
    if (i < n) {
#pragma unroll 4
        for (int j = tid >> 6; j < n; j += NT / 64) {
            A[i + (long)j * lda] = i >= j ? S[i + j * SLD] : 0.0;
            if (kInv) inv[i + (long)j * ldinv] = i >= j ? X[i + j * SLD] : 0.0;
        }
    }
    __syncthreads();
    if (tid == 0 && logdet) *logdet = 2.0 * (sm.red[0] + sm.red[1]);
    const int flag = sm.flag;
    __syncthreads();  // the shared memory is free again
    return flag;
}

__device__ inline int potrf_small(int n, double* A, long lda, LaSmem<double>& sm, double* logdet, double* inv,
                                  long ldinv) {
    const int tid = threadIdx.x;
    double* S = &sm.A[0][0];  // 64 x 68 (fits in the operand tile buffers)
    const int N = (n + 7) & ~7;
    {
        // every load issued before the first store (16 columns per thread)
        const int i = tid & 63, j0 = tid >> 6;
        double v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int j = j0 + 4 * q;
            v[q] = (i < n && j < n) ? A[i + (long)j * lda] : (i == j ? 1.0 : 0.0);
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int j = j0 + 4 * q;
            if (i < N && j < N) S[i + j * SLD] = v[q];
        }
    }
    __syncthreads();
    return inv ? potrf_finish<true, LaSmem<double>>(n, A, lda, logdet, inv, ldinv)
               : potrf_finish<false, LaSmem<double>>(n, A, lda, logdet, inv, ldinv);
}

// FP64 Cholesky with the inverse of the factor for 64 < n <= 128, as a 2 x 2
// block factorization around potrf_small (64 + n2 with n2 = n - 64):
//   L11 = chol(A11), X11 = L11^{-1};  L21 = A21 X11^T;  A22 -= L21 L21^T;
//   L22 = chol(A22), X22 = L22^{-1};  X21 = -X22 (L21 X11)
// so that everything but the two diagonal factorizations runs as products on
// the tensor pipe.  A and inv get zeros above the diagonal.  Returns 0 or the
// 1-based index of the first bad pivot; logdet (thread 0) = 2 sum log L_ii.
__device__ inline int potrf_mid(int n, double* A, long lda, LaSmem<double>& sm, double* logdet, double* inv,
                                long ldinv) {
    const int n2 = n - 64;
    double ld1 = 0.0, ld2 = 0.0;
    const int info1 = potrf_small(64, A, lda, sm, &ld1, inv, ldinv);
    double* A21 = A + 64;
    double* A22 = A + 64 + 64 * lda;
    double* X21 = inv + 64;
    double* X22 = inv + 64 + 64 * ldinv;
    // L21 = A21 X11^T in place (a single output tile reads all of A21 first)
    gemm<double, false, true, true>(n2, 64, 64, 1.0, A21, lda, inv, ldinv, 0.0, A21, lda, sm);
    gemm<double, false, true>(n2, n2, 64, -1.0, A21, lda, A21, lda, 1.0, A22, lda, sm);
    const int info2 = potrf_small(n2, A22, lda, sm, &ld2, X22, ldinv);
    gemm<double, false, false>(n2, 64, 64, 1.0, A21, lda, inv, ldinv, 0.0, X21, ldinv, sm);
    gemm<double, false, false, true>(n2, 64, n2, -1.0, X22, ldinv, X21, ldinv, 0.0, X21, ldinv, sm);
    for (int e = threadIdx.x; e < 64 * n2; e += kThreads) {
        const int i = e & 63, j = 64 + (e >> 6);
        A[i + (long)j * lda] = 0.0;
        inv[i + (long)j * ldinv] = 0.0;
    }
    __syncthreads();
    if (threadIdx.x == 0 && logdet) *logdet = ld1 + ld2;
    return info1 ? info1 : (info2 ? info2 + 64 : 0);
}

// The scheme of potrf_core for 64 < n <= 128 with the inverse, by 256 threads, one
// CTA per SM: L and X = L^{-1} share one array, X transposed above the diagonal
// blocks (its own diagonal blocks beside it), so that block column k holds X's block
// row k in the rows above and L's panel below, and one form of tile update,
//   C(p, q) -= panel(p) panel(q)^T,  q > k, p <= k (X) or p >= q (L),
// serves both.  A launch of one 100 x 100 factorization 70 -> 46 us against potrf_mid's
// two factorizations with products through memory between them.
constexpr int SLD2 = 132;
struct Potrf128Smem {
    double S[128 * SLD2];
    double XD[16][64];  // diagonal blocks of X, column-major
    double red[kThreads / 32];
    int flag;
};

static __device__ __noinline__ int potrf_128(int n, double* A, long lda, double* logdet, double* inv, long ldinv) {
    extern __shared__ __align__(16) unsigned char la_dyn_smem[];
    Potrf128Smem& sm = *reinterpret_cast<Potrf128Smem*>(la_dyn_smem);
    double* S = sm.S;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int nbk = (n + 7) >> 3, N = nbk << 3;
    {
        const int i = tid & 127;
        for (int j0 = tid >> 7; j0 < N; j0 += 16) {  // eight loads in flight
            double v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int j = j0 + 2 * q;
                v[q] = (i < n && j <= i && j < n) ? A[i + (long)j * lda] : (i == j ? 1.0 : 0.0);
            }
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (i < N && j0 + 2 * q < N) S[i + (j0 + 2 * q) * SLD2] = v[q];
        }
    }
    __syncthreads();
    int bad = 0;
    for (int k = 0; k < nbk; ++k) {
        const int k0 = k << 3;
        const int row = k0 + tid, c = tid - 128;
        const bool prow = tid < 128 && row < N, pcol = tid >= 128 && c < k0;
        double* base = (tid < 128 ? S + row : S + c) + k0 * SLD2;  // a row of L's panel, or of X's block row transposed
        double l[36], x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j <= i; ++j) l[i * (i + 1) / 2 + j] = S[(k0 + i) + (k0 + j) * SLD2];
        const int e = c - k0;  // column of X's diagonal block
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = prow || pcol ? base[j * SLD2] : (tid >= 128 && e == j ? 1.0 : 0.0);
        __syncthreads();  // the block is read before its rows are rewritten
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const double d = l[j * (j + 1) / 2 + j];
            if (!(d > 0.0) && bad == 0 && k0 + j < n) bad = k0 + j + 1;
            const double r = rsqrt(d);
#pragma unroll
            for (int i = j + 1; i < 8; ++i) l[i * (i + 1) / 2 + j] *= r;
            x[j] *= r;
#pragma unroll
            for (int i = j + 1; i < 8; ++i) {
#pragma unroll
                for (int q = j + 1; q <= i; ++q)
                    l[i * (i + 1) / 2 + q] = fma(-l[i * (i + 1) / 2 + j], l[q * (q + 1) / 2 + j], l[i * (i + 1) / 2 + q]);
                x[i] = fma(-l[i * (i + 1) / 2 + j], x[j], x[i]);
            }
        }
        if (prow || pcol) {
#pragma unroll
            for (int j = 0; j < 8; ++j) base[j * SLD2] = tid < 128 && j > tid ? 0.0 : x[j];
        } else if (tid >= 128 && e >= 0 && e < 8) {
#pragma unroll
            for (int j = 0; j < 8; ++j) sm.XD[k][j + 8 * e] = x[j];
        }
        __syncthreads();
        for (int q = k + 1 + w; q < nbk; q += kThreads / 32) {
            const double* P = S + (k0 + t) * SLD2 + g;  // panel(p): rows 8 p + g
            const double b0 = P[8 * q], b1 = P[8 * q + 4 * SLD2];
            double* C = S + g + (8 * q + 2 * t) * SLD2;
            auto tile = [&](int p, double a0, double a1) {
                double acc[2] = {-C[8 * p], -C[8 * p + SLD2]};
                mma_f64(acc, a0, b0);
                mma_f64(acc, a1, b1);
                C[8 * p] = -acc[0];
                C[8 * p + SLD2] = -acc[1];
            };
#pragma unroll 4
            for (int p = 0; p < k; ++p) tile(p, P[8 * p], P[8 * p + 4 * SLD2]);
            tile(k, sm.XD[k][t + 8 * g], sm.XD[k][t + 4 + 8 * g]);
#pragma unroll 4
            for (int p = q; p < nbk; ++p) tile(p, P[8 * p], P[8 * p + 4 * SLD2]);
        }
        __syncthreads();
    }
    double part = tid < n ? log(S[tid + tid * SLD2]) : 0.0;
    for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
    if (lane == 0) sm.red[w] = part;
    if (tid == 0) sm.flag = bad;
    for (int j = w; j < n; j += kThreads / 32)
        for (int i = lane; i < n; i += 32) {
            A[i + (long)j * lda] = i >= j ? S[i + j * SLD2] : 0.0;
            inv[i + (long)j * ldinv] = i < j ? 0.0 : ((i >> 3) == (j >> 3) ? sm.XD[i >> 3][(i & 7) + 8 * (j & 7)] : S[j + i * SLD2]);
        }
    __syncthreads();
    if (tid == 0 && logdet) *logdet = 2.0 * ((sm.red[0] + sm.red[1]) + (sm.red[2] + sm.red[3]));
    const int flag = sm.flag;
    __syncthreads();
    return flag;
}

// In-place lower Cholesky (see potrf_blocked); FP64 matrices up to 64 go
// through potrf_small, and up to 128 through potrf_mid when the inverse is
// asked for.  With `inv`, L^{-1} is also written there (ld ldinv).
template <typename T>
__device__ inline int potrf_lower(int n, T* A, long lda, LaSmem<T>& sm, double* logdet, T* inv = nullptr,
                                  long ldinv = 0) {
    if constexpr (sizeof(T) == 8) {
        if (n <= 64) return potrf_small(n, A, lda, sm, logdet, inv, ldinv);
        if (n <= 128 && inv) return potrf_mid(n, A, lda, sm, logdet, inv, ldinv);
    }
    const int info = potrf_blocked(n, A, lda, sm, logdet);
    if (inv) {
        for (long e = threadIdx.x; e < (long)n * n; e += kThreads) {
            const int i = (int)(e % n), j = (int)(e / n);
            inv[i + (long)j * ldinv] = i == j ? (T)1 : (T)0;
        }
        __syncthreads();
        trsm_left_lower<T>(n, n, A, lda, inv, ldinv, sm);
    }
    return info;
}

}  // namespace mra
