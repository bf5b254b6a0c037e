// MLP surrogate of the MRA log-likelihood: n_in -> 128 -> 128 -> 1 with SiLU,
// BF16 weights in the forward and backward passes, FP32 accumulation, FP32
// master parameters updated by Adam (include/mra_surrogate.h).
//
// One kernel does the forward pass, the backward pass and the per-CTA
// gradient sums over a grid-strided set of 16-sample tiles; a second kernel
// adds the per-CTA sums in a fixed order (deterministic) and applies Adam.
// Predictions without input gradients (the screening of candidate parameter
// vectors) run k_mlp_forward_tc instead, whose 128 x 128 layer is a
// tcgen05.mma product in tensor memory.
// Four threads of a CTA share hidden unit h, each a quarter of the tile's
// samples; W2 sits in shared memory in BF16 with padded rows, read along row h in the
// forward product and column-wise in the backward one, both free of bank conflicts.  The passes are
// chains of dependent sums of fixed order, a few tiles at most in flight, so what
// counts is how many of them run side by side: with one thread per hidden unit
// and 16 samples each a training step of 160 samples took 48 us, now 12, and the
// gradients of 64 samples 55 us, now 9 (4-sample tiles); every sum keeps its order,
// so the results are bitwise the same.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "../../include/mra_surrogate.h"
#include "mra_kernels.cuh"

namespace {

constexpr int H = 128;     // hidden width
constexpr int S = 16;      // samples per training tile
constexpr int SQ = 4;      // samples per tile of a small prediction
constexpr int NT = 4 * H;  // threads of a pass
constexpr int MAXD = 64;   // largest input width
constexpr long MAXN = 65536;

struct Layout {
    long W1, b1, W2, b2, w3, b3, P;
    explicit Layout(int D) {
        W1 = 0;
        b1 = W1 + (long)H * D;
        W2 = b1 + H;
        b2 = W2 + (long)H * H;
        w3 = b2 + H;
        b3 = w3 + H;
        P = b3 + 1;
    }
};

struct MlpArgs {
    int D;
    long N;
    long W1, b1, W2, b2, w3, b3, P;
    const float* master;
    const __nv_bfloat16* W1b;   // [H][D]
    const __nv_bfloat16* W2b;   // [H][H]
    const __nv_bfloat16* w3b;   // [H]
    const float* X;             // [N][D]
    const float* T;             // [N]      (TRAIN)
    float* partial;             // [grid][P+1] per-CTA gradient sums, last = loss sum (TRAIN)
    float* Y;                   // [N]      (PREDICT*)
    float* G;                   // [N][D]   (PREDICT_GRAD)
};

__device__ __forceinline__ float sigm(float z) { return 1.0f / (1.0f + expf(-z)); }

// 4-byte asynchronous global -> shared copies: every load of a prologue in flight at once
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

constexpr int WS = H + 2;  // row stride of W2 and of W1 transposed: consecutive rows fall on different banks

size_t smem_bytes(int D, int ns) {
    return (size_t)H * WS * sizeof(__nv_bfloat16)        // W2 (row-major)
           + (((size_t)D * WS * sizeof(__nv_bfloat16) + 15) & ~(size_t)15)  // W1 transposed [d][h]
           + (size_t)ns * MAXD * sizeof(float)           // x tile
           + 3 * (size_t)ns * H * sizeof(float)          // a1, g_z2, g_z1 tiles
           + (size_t)ns * 4 * sizeof(float);             // y partial sums per warp
}

// ST: samples per tile; thread (h, sg) handles hidden unit h of samples sg ST/4 ...
template <int ST>
__global__ void __launch_bounds__(NT, 1) k_mlp_pass(MlpArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int PT = ST / 4;
    const int D = a.D;
    const int tid = threadIdx.x, h = tid & (H - 1), sg = tid >> 7, warp = (tid >> 5) & 3, lane = tid & 31;
    __nv_bfloat16* W2s = reinterpret_cast<__nv_bfloat16*>(smem);
    __nv_bfloat16* W1t = W2s + H * WS;
    float* xs = reinterpret_cast<float*>(smem + (size_t)H * WS * 2 + (((size_t)D * WS * 2 + 15) & ~(size_t)15));
    float* a1s = xs + ST * MAXD;
    float* gzs = a1s + ST * H;
    float* g1s = gzs + ST * H;
    float* red = g1s + ST * H;

#pragma unroll
    for (int q = 0; q < H * H / 2 / NT; ++q) {
        const int e = tid + q * NT;
        cp_async4(reinterpret_cast<unsigned*>(W2s) + (e >> 6) * (WS / 2) + (e & 63),
                  reinterpret_cast<const unsigned*>(a.W2b) + e);
    }
    // the first tile's inputs with the weights; the next tiles' at the end of the loop
    auto load_x = [&](long tile) {
        for (int d = lane; d < D; d += 32)
            for (int s = tid >> 5; s < ST; s += NT / 32) {
                const long i = tile * ST + s;
                if (i < a.N) cp_async4(xs + s * MAXD + d, a.X + i * D + d);
                else xs[s * MAXD + d] = 0.f;
            }
    };
    load_x(blockIdx.x);
    {
        __nv_bfloat16 v[MAXD / 4];
#pragma unroll
        for (int q = 0; q < MAXD / 4; ++q)
            if (sg + 4 * q < D) v[q] = a.W1b[h * D + sg + 4 * q];
#pragma unroll
        for (int q = 0; q < MAXD / 4; ++q)
            if (sg + 4 * q < D) W1t[(sg + 4 * q) * WS + h] = v[q];
    }
    const float b1h = a.master[a.b1 + h], b2h = a.master[a.b2 + h], b3 = a.master[a.b3];
    const float w3h = __bfloat162float(a.w3b[h]);
    const long ntiles = (a.N + ST - 1) / ST;
    for (long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long s0 = tile * ST;
        const int ns = (int)min((long)ST, a.N - s0);
        cp_async_all();
        __syncthreads();
        // layer 1
        float z1[PT], z2[PT];
#pragma unroll
        for (int j = 0; j < PT; ++j) z1[j] = b1h;
#pragma unroll 4
        for (int d = 0; d < D; ++d) {
            const float w = __bfloat162float(W1t[d * WS + h]);
#pragma unroll
            for (int j = 0; j < PT; ++j) z1[j] = fmaf(w, xs[(sg * PT + j) * MAXD + d], z1[j]);
        }
#pragma unroll
        for (int j = 0; j < PT; ++j) a1s[(sg * PT + j) * H + h] = z1[j] * sigm(z1[j]);
        __syncthreads();
        // layer 2 and the output
#pragma unroll
        for (int j = 0; j < PT; ++j) z2[j] = b2h;
        const float4* ar = reinterpret_cast<const float4*>(a1s + sg * PT * H);
        const __nv_bfloat162* w2r = reinterpret_cast<const __nv_bfloat162*>(W2s + h * WS);
#pragma unroll 8
        for (int q = 0; q < H / 4; ++q) {
            const float2 w0 = __bfloat1622float2(w2r[2 * q]), w1 = __bfloat1622float2(w2r[2 * q + 1]);
#pragma unroll
            for (int j = 0; j < PT; ++j) {
                const float4 x = ar[j * (H / 4) + q];
                z2[j] = fmaf(w0.x, x.x, z2[j]);
                z2[j] = fmaf(w0.y, x.y, z2[j]);
                z2[j] = fmaf(w1.x, x.z, z2[j]);
                z2[j] = fmaf(w1.y, x.w, z2[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            float p = w3h * (z2[j] * sigm(z2[j]));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
            if (lane == 0) red[(sg * PT + j) * 4 + warp] = p;
        }
        __syncthreads();
        // output errors and the backward step through the output layer
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            const int s = sg * PT + j;
            const float y = b3 + ((red[s * 4 + 0] + red[s * 4 + 1]) + (red[s * 4 + 2] + red[s * 4 + 3]));
            const float gy = s < ns ? 1.f : 0.f;
            if (h == 0 && s < ns) a.Y[s0 + s] = y;
            const float sg2 = sigm(z2[j]);
            gzs[s * H + h] = gy * w3h * (sg2 * (1.f + z2[j] * (1.f - sg2)));
        }
        __syncthreads();
        // through W2 and the first activation
        float gz1[PT];
#pragma unroll
        for (int j = 0; j < PT; ++j) gz1[j] = 0.f;
#pragma unroll 4
        for (int o = 0; o < H; o += 4) {
            float w[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) w[u] = __bfloat162float(W2s[(o + u) * WS + h]);
#pragma unroll
            for (int j = 0; j < PT; ++j) {
                const float4 gz = *reinterpret_cast<const float4*>(gzs + (sg * PT + j) * H + o);
                gz1[j] = fmaf(w[0], gz.x, gz1[j]);
                gz1[j] = fmaf(w[1], gz.y, gz1[j]);
                gz1[j] = fmaf(w[2], gz.z, gz1[j]);
                gz1[j] = fmaf(w[3], gz.w, gz1[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            const float sg1 = sigm(z1[j]);
            gz1[j] *= sg1 * (1.f + z1[j] * (1.f - sg1));
            g1s[(sg * PT + j) * H + h] = gz1[j];
        }
        __syncthreads();
        {
            // d y / d x: sum over hidden units of W1[h][d] g_z1[h]
            for (int e = tid; e < ST * D; e += NT) {
                int s = e / D, d = e % D;
                float acc = 0.f;
#pragma unroll 8
                for (int k = 0; k < H; ++k) acc = fmaf(__bfloat162float(W1t[d * WS + k]), g1s[s * H + k], acc);
                if (s < ns) a.G[(s0 + s) * D + d] = acc;
            }
        }
        __syncthreads();
        if (tile + gridDim.x < ntiles) load_x(tile + gridDim.x);
    }
}

// ---------------------------------------------------------------------------
// training pass
// ---------------------------------------------------------------------------
// A cluster of four CTAs takes a tile of 16 samples: each CTA runs the forward and
// backward chains of four of them, one sample and hidden unit per thread, writes
// what the weight gradients need (a1, g_z2, a2, g_z1, x, g_y) to all four, and then
// sums a quarter of the weights' gradients over the 16 samples.  The chains are
// latency: with them spread over four CTAs, and the launches overlapped, a step of 160
// samples takes 12 us instead of 23 with one CTA per tile, and the order of every sum
// is the same.
// Launched with programmatic serialization: the inputs, which no step changes, load
// while the previous step's Adam kernel runs.
struct TrainSmem {
    __nv_bfloat16 W2[H * WS];   // row-major
    __nv_bfloat16 W1t[MAXD * WS];
    float x[S * MAXD], a1[S * H], gz[S * H], a2[S * H], g1[S * H];
    float red[S / 4 * 4], gy[S], err[S];
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// v to the same shared address in each CTA of the cluster
__device__ __forceinline__ void store_all(float* p, float v) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        unsigned q;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(q) : "r"(a), "r"(r));
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(q), "f"(v) : "memory");
    }
}

__global__ void __cluster_dims__(4, 1, 1) __launch_bounds__(NT, 1) k_mlp_train(MlpArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    TrainSmem& sm = *reinterpret_cast<TrainSmem*>(smem);
    constexpr int SC = S / 4;  // samples of this CTA, one per thread group
    const int D = a.D, cr = (int)cluster_rank();
    const int tid = threadIdx.x, h = tid & (H - 1), sg = tid >> 7, warp = (tid >> 5) & 3, lane = tid & 31;
    const int smp = cr * SC + sg;  // this thread's sample of the tile
    const long ntiles = (a.N + S - 1) / S, n_cl = gridDim.x / 4;
    // the tile's inputs: all 16 samples (the gradients of W1 read them)
    auto load_x = [&](long tile) {
        for (int d = lane; d < D; d += 32)
            for (int s = tid >> 5; s < S; s += NT / 32) {
                const long i = tile * S + s;
                if (i < a.N) cp_async4(sm.x + s * MAXD + d, a.X + i * D + d);
                else sm.x[s * MAXD + d] = 0.f;
            }
    };
    const long tile0 = blockIdx.x / 4;
    load_x(tile0);
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the weights of the previous step
#pragma unroll
    for (int q = 0; q < H * H / 2 / NT; ++q) {
        const int e = tid + q * NT;
        cp_async4(reinterpret_cast<unsigned*>(sm.W2) + (e >> 6) * (WS / 2) + (e & 63),
                  reinterpret_cast<const unsigned*>(a.W2b) + e);
    }
    {
        __nv_bfloat16 v[MAXD / 4];
#pragma unroll
        for (int q = 0; q < MAXD / 4; ++q)
            if (sg + 4 * q < D) v[q] = a.W1b[h * D + sg + 4 * q];
#pragma unroll
        for (int q = 0; q < MAXD / 4; ++q)
            if (sg + 4 * q < D) sm.W1t[(sg + 4 * q) * WS + h] = v[q];
    }
    const float b1h = a.master[a.b1 + h], b2h = a.master[a.b2 + h], b3 = a.master[a.b3];
    const float w3h = __bfloat162float(a.w3b[h]);
    float db = 0.f, db3 = 0.f, lsum = 0.f;  // db: of b1 (sg 2), b2 (sg 1) or w3 (sg 0), on the CTA of that rank
    // dW2[32 cr + 8 sg + q][h], dW1[4 (4 q + sg) + cr][h]
    float dW2[H / 16], dW1[MAXD / 16];
#pragma unroll
    for (int q = 0; q < H / 16; ++q) dW2[q] = 0.f;
#pragma unroll
    for (int q = 0; q < MAXD / 16; ++q) dW1[q] = 0.f;

    cluster_sync();  // every CTA of the cluster runs before any writes to it
    for (long tile = tile0; tile < ntiles; tile += n_cl) {
        const long s0 = tile * S;
        const bool valid = s0 + smp < a.N;
        const float tgt = valid ? a.T[s0 + smp] : 0.f;
        cp_async_all();
        __syncthreads();
        // layer 1
        float z1 = b1h;
#pragma unroll 4
        for (int d = 0; d < D; ++d) z1 = fmaf(__bfloat162float(sm.W1t[d * WS + h]), sm.x[smp * MAXD + d], z1);
        const float s1 = sigm(z1), a1 = z1 * s1;
        store_all(sm.a1 + smp * H + h, a1);
        __syncthreads();
        // layer 2 and the output
        float z2 = b2h;
        const __nv_bfloat162* w2r = reinterpret_cast<const __nv_bfloat162*>(sm.W2 + h * WS);
        const float4* ar = reinterpret_cast<const float4*>(sm.a1 + smp * H);
#pragma unroll 8
        for (int q = 0; q < H / 4; ++q) {
            const float2 w0 = __bfloat1622float2(w2r[2 * q]), w1 = __bfloat1622float2(w2r[2 * q + 1]);
            const float4 x = ar[q];
            z2 = fmaf(w0.x, x.x, z2);
            z2 = fmaf(w0.y, x.y, z2);
            z2 = fmaf(w1.x, x.z, z2);
            z2 = fmaf(w1.y, x.w, z2);
        }
        const float s2 = sigm(z2), a2 = z2 * s2;
        {
            float p = w3h * a2;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
            if (lane == 0) sm.red[sg * 4 + warp] = p;
        }
        __syncthreads();
        // output error and the backward step through the output layer
        const float y = b3 + ((sm.red[sg * 4 + 0] + sm.red[sg * 4 + 1]) + (sm.red[sg * 4 + 2] + sm.red[sg * 4 + 3]));
        const float e = valid ? y - tgt : 0.f;
        const float gy = 2.f * e / (float)a.N;
        store_all(sm.gz + smp * H + h, gy * w3h * (s2 * (1.f + z2 * (1.f - s2))));
        store_all(sm.a2 + smp * H + h, a2);
        if (h == 0) {
            store_all(sm.gy + smp, gy);
            store_all(sm.err + smp, e);
        }
        __syncthreads();
        // through W2 and the first activation
        float gz1 = 0.f;
#pragma unroll 8
        for (int o = 0; o < H; o += 4) {
            const float4 gz = *reinterpret_cast<const float4*>(sm.gz + smp * H + o);
            gz1 = fmaf(__bfloat162float(sm.W2[(o + 0) * WS + h]), gz.x, gz1);
            gz1 = fmaf(__bfloat162float(sm.W2[(o + 1) * WS + h]), gz.y, gz1);
            gz1 = fmaf(__bfloat162float(sm.W2[(o + 2) * WS + h]), gz.z, gz1);
            gz1 = fmaf(__bfloat162float(sm.W2[(o + 3) * WS + h]), gz.w, gz1);
        }
        gz1 *= s1 * (1.f + z1 * (1.f - s1));
        store_all(sm.g1 + smp * H + h, gz1);
        cluster_sync();  // the 16 samples of the tile are in every CTA
        {
            float v[S];
#pragma unroll
            for (int s = 0; s < S; ++s) v[s] = sm.a1[s * H + h];
#pragma unroll
            for (int q = 0; q < H / 16; q += 4) {
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const float4 gz = *reinterpret_cast<const float4*>(sm.gz + s * H + 32 * cr + 8 * sg + q);
                    acc[0] = fmaf(gz.x, v[s], acc[0]);
                    acc[1] = fmaf(gz.y, v[s], acc[1]);
                    acc[2] = fmaf(gz.z, v[s], acc[2]);
                    acc[3] = fmaf(gz.w, v[s], acc[3]);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) dW2[q + u] += acc[u];
            }
#pragma unroll
            for (int s = 0; s < S; ++s) v[s] = sm.g1[s * H + h];
#pragma unroll
            for (int q = 0; q < MAXD / 16; ++q) {
                const int d = 4 * (4 * q + sg) + cr;
                if (d >= D) break;
                float acc = 0.f;
#pragma unroll
                for (int s = 0; s < S; ++s) acc = fmaf(v[s], sm.x[s * MAXD + d], acc);
                dW1[q] += acc;
            }
            if (sg == cr) {
                if (sg == 0) {
#pragma unroll
                    for (int s = 0; s < S; ++s) db = fmaf(sm.gy[s], sm.a2[s * H + h], db);
                } else if (sg == 1) {
#pragma unroll
                    for (int s = 0; s < S; ++s) db += sm.gz[s * H + h];
                } else if (sg == 2) {
#pragma unroll
                    for (int s = 0; s < S; ++s) db += v[s];
                } else if (h == 0) {
                    for (int s = 0; s < S; ++s) {
                        lsum += sm.err[s] * sm.err[s];
                        db3 += sm.gy[s];
                    }
                }
            }
        }
        cluster_sync();  // no CTA's tile is overwritten, and none exits, while another may write to it
        if (tile + n_cl < ntiles) load_x(tile + n_cl);
    }
    float* out = a.partial + tile0 * (a.P + 1);
#pragma unroll
    for (int q = 0; q < MAXD / 16; ++q) {
        const int d = 4 * (4 * q + sg) + cr;
        if (d < D) out[a.W1 + (long)h * D + d] = dW1[q];
    }
#pragma unroll
    for (int q = 0; q < H / 16; ++q) out[a.W2 + (long)(32 * cr + 8 * sg + q) * H + h] = dW2[q];
    if (sg == cr) {
        if (sg == 0) out[a.w3 + h] = db;
        if (sg == 1) out[a.b2 + h] = db;
        if (sg == 2) out[a.b1 + h] = db;
        if (sg == 3 && h == 0) {
            out[a.b3] = db3;
            out[a.P] = lsum;
        }
    }
}

// Sums the per-CTA partials in CTA order; grad_out != nullptr: store the
// gradient (and loss); else one Adam step on the master weights and their BF16
// copies.  bc1/bc2: 1 - beta^t bias corrections.
__global__ void k_mlp_reduce_adam(long P, int nblk, const float* __restrict__ partial, float* grad_out,
                                  float* loss_out, float* master, float* m, float* v, __nv_bfloat16* W1b,
                                  __nv_bfloat16* W2b, __nv_bfloat16* w3b, long oW2, long ob2, long ow3, long ob3,
                                  long ob1, float lr, float bc1, float bc2) {
    long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the pass's sums
    if (p > P) return;
    float g = 0.f;
#pragma unroll 8
    for (int c = 0; c < nblk; ++c) g += partial[(long)c * (P + 1) + p];
    if (p == P) {
        if (loss_out) *loss_out = g;
        return;
    }
    if (grad_out) {
        grad_out[p] = g;
        return;
    }
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    float mm = b1 * m[p] + (1.f - b1) * g;
    float vv = b2 * v[p] + (1.f - b2) * g * g;
    m[p] = mm;
    v[p] = vv;
    float w = master[p] - lr * (mm / bc1) / (sqrtf(vv / bc2) + eps);
    master[p] = w;
    if (p < ob1) W1b[p] = __float2bfloat16_rn(w);
    else if (p >= oW2 && p < ob2) W2b[p - oW2] = __float2bfloat16_rn(w);
    else if (p >= ow3 && p < ob3) w3b[p - ow3] = __float2bfloat16_rn(w);
}

__global__ void k_mlp_sync_bf16(long P, const float* master, __nv_bfloat16* W1b, __nv_bfloat16* W2b,
                                __nv_bfloat16* w3b, long oW2, long ob2, long ow3, long ob3, long ob1) {
    long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    float w = master[p];
    if (p < ob1) W1b[p] = __float2bfloat16_rn(w);
    else if (p >= oW2 && p < ob2) W2b[p - oW2] = __float2bfloat16_rn(w);
    else if (p >= ow3 && p < ob3) w3b[p - ow3] = __float2bfloat16_rn(w);
}

// ---------------------------------------------------------------------------
// Forward pass on the 5th-generation tensor cores (prediction without input
// gradients).  One CTA of 512 threads takes a tile of 128 samples (sample s = TMEM
// lane s), four threads per sample, each a quarter of the hidden units:
//   layer 1 (n_in x 128, small) on the FP32 cores, exactly as k_mlp_pass;
//   layer 2 (128 x 128 x 128) as tcgen05.mma kind::tf32 with the product in
//     tensor memory: a1 is split into a TF32 high part and the FP32 remainder
//     (a1 = hi + lo, hi exact in TF32), W2 is BF16 and hence exact in TF32, so
//     hi W2^T + lo W2^T is FP32-accurate (the remainder's own truncation to TF32
//     costs at most 2^-21 |a1|);
//   the output layer on the FP32 cores from the product read back by tcgen05.ld.
// The FP32 parts (layer 1 and 256 SiLUs per sample) set the time: 65,536 samples in one
// launch took 140 us with one thread per sample and 50 with four (mra_mlp_predict
// launches them in runs of a tile per SM, behind their input copies).
// Operands sit in shared memory in the canonical K-major layout without
// swizzle: 8-row x 16-byte core matrices, the two core matrices of one MMA's K
// slice 128 bytes apart (leading byte offset), consecutive 8-row groups 4096
// bytes apart (stride byte offset).  One thread issues the MMAs and commits
// them to an mbarrier; the others wait on it with a bounded spin.
constexpr int TC_M = 128;                    // samples per tile = MMA M = TMEM lanes
constexpr unsigned TC_LBO = 128, TC_SBO = 4096;
constexpr int TC_T = 4 * TC_M;               // threads of the CTA
constexpr long kTcSpin = 1L << 24;           // bounded waits (about a second)

struct TcSmem {
    float Ahi[TC_M * H];                     // 64 KB each, canonical K-major layout; after the product the output sums
                                             // of each quarter of the hidden units [4][sample]
    float Alo[TC_M * H];                     // first the tile's inputs [sample][n_in | 1]
    float W2f[H * H];                        // rows = output units
    float W1t[MAXD * H];                     // layer 1 weights [d][h]
    float b1[H], b2[H], w3[H];
    unsigned long long bar;                  // MMA completion
    unsigned tmem_base;
};

// element (row, k) of a 128-row, 128-deep K-major tile of 4-byte elements
__device__ __forceinline__ int tc_idx(int row, int k) {
    return (row >> 3) * (int)(TC_SBO / 4) + (k >> 2) * (int)(TC_LBO / 4) + (row & 7) * 4 + (k & 3);
}
__device__ __forceinline__ unsigned tc_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// shared-memory matrix descriptor: start, leading / stride byte offsets (>> 4),
// descriptor version 1 (bits 46-47), no swizzle
__device__ __forceinline__ unsigned long long tc_desc(unsigned addr) {
    return (unsigned long long)((addr >> 4) & 0x3FFF) | ((unsigned long long)((TC_LBO >> 4) & 0x3FFF) << 16) |
           ((unsigned long long)((TC_SBO >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
// instruction descriptor: D F32 (bits 4-5 = 1), A and B TF32 (bits 7-9, 10-12 = 2),
// both K-major, N = 128 (bits 17-22 = N >> 3), M = 128 (bits 24-28 = M >> 4)
constexpr unsigned kTcIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(H >> 3) << 17) | ((unsigned)(TC_M >> 4) << 24);

// D[tmem] (+)= A B^T for one K slice of 8, A and B given by their descriptors
__device__ __forceinline__ void tc_mma(unsigned tmem, unsigned long long adesc, unsigned long long bdesc, bool acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
        "l"(adesc), "l"(bdesc), "r"(kTcIdesc), "r"((unsigned)acc)
        : "memory");
}
__device__ __forceinline__ bool tc_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(tc_smem(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// 32 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tc_ld32(unsigned taddr, float (&v)[32]) {
    unsigned r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int q = 0; q < 32; ++q) v[q] = __uint_as_float(r[q]);
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// z[0..1] += a * b, two FP32 multiply-adds in one instruction
__device__ __forceinline__ void fma2(float* z, float2 a, float2 b) {
    float2 c = make_float2(z[0], z[1]);
    unsigned long long& cc = *reinterpret_cast<unsigned long long*>(&c);
    asm("fma.rn.f32x2 %0, %1, %2, %0;"
        : "+l"(cc)
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    z[0] = c.x;
    z[1] = c.y;
}

// y = MLP(x) for a.N samples (a.Y), one tile per CTA; *err = 1 if a bounded wait gave up.
__global__ void __launch_bounds__(TC_T, 1) k_mlp_forward_tc(MlpArgs a, int* err) {
    extern __shared__ __align__(1024) unsigned char tc_raw[];
    TcSmem& sm = *reinterpret_cast<TcSmem*>(tc_raw);
    const int tid = threadIdx.x, warp = tid >> 5, D = a.D;
    const int smp = tid & (TC_M - 1), hq = tid / TC_M;  // sample of the tile, quarter of the hidden units
    const int XD = D | 1;
    const long s0 = (long)blockIdx.x * TC_M;
    const bool valid = s0 + smp < a.N;
    {
        const long left = a.N - s0;
        const int n = (int)(left < TC_M ? left : TC_M) * D;
        const float* X = a.X + s0 * D;
        for (int e = tid; e < TC_M * D; e += TC_T) {
            const int q = e / D;
            float* dst = sm.Alo + e + q * (XD - D);
            if (e < n) cp_async4(dst, X + e);
            else *dst = 0.f;
        }
    }
    {
        uint4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = reinterpret_cast<const uint4*>(a.W2b)[tid + q * TC_T];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = 8 * (tid + q * TC_T);
            const unsigned u[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[2 * x]));
                const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[2 * x + 1]));
                *reinterpret_cast<float4*>(sm.W2f + tc_idx(e / H, e % H + 4 * x)) = make_float4(lo.x, lo.y, hi.x, hi.y);
            }
        }
        __nv_bfloat16 w[MAXD / 4];
#pragma unroll
        for (int q = 0; q < MAXD / 4; ++q)
            if (hq + 4 * q < D) w[q] = a.W1b[smp * D + hq + 4 * q];
#pragma unroll
        for (int q = 0; q < MAXD / 4; ++q)
            if (hq + 4 * q < D) sm.W1t[(hq + 4 * q) * H + smp] = __bfloat162float(w[q]);
    }
    for (int h = tid; h < H; h += TC_T) {
        sm.b1[h] = a.master[a.b1 + h];
        sm.b2[h] = a.master[a.b2 + h];
        sm.w3[h] = __bfloat162float(a.w3b[h]);
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(tc_smem(&sm.bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        // 128 TMEM columns: the 128 x 128 FP32 product of one tile
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem(&sm.tmem_base)),
                     "r"(H)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = sm.tmem_base;
    const unsigned lane_addr = tmem + ((unsigned)((warp & 3) * 32) << 16) + (unsigned)(32 * hq);
    const float b3 = a.master[a.b3];
    const float* xs = sm.Alo;
    cp_async_all();
    __syncthreads();
    // layer 1 on the FP32 cores, in k_mlp_pass's order: z1 = b1 + sum_d W1[h][d] x[d]
    float z[H / 4];
#pragma unroll
    for (int h = 0; h < H / 4; ++h) z[h] = sm.b1[32 * hq + h];
    for (int d = 0; d < D; ++d) {
        const float xd = xs[smp * XD + d];
        const float2 x2 = make_float2(xd, xd);
        const float4* wr = reinterpret_cast<const float4*>(sm.W1t + d * H + 32 * hq);
#pragma unroll
        for (int q = 0; q < H / 16; ++q) {
            const float4 w = wr[q];
            fma2(z + 4 * q, make_float2(w.x, w.y), x2);
            fma2(z + 4 * q + 2, make_float2(w.z, w.w), x2);
        }
    }
    __syncthreads();  // the inputs have been read
#pragma unroll
    for (int h = 0; h < H / 4; h += 4) {
        float4 hi, lo;
        float* ph = &hi.x;
        float* pl = &lo.x;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float a1 = z[h + e] * sigm(z[h + e]);
            ph[e] = __uint_as_float(__float_as_uint(a1) & 0xffffe000u);  // exact in TF32
            pl[e] = a1 - ph[e];
        }
        const int at = tc_idx(smp, 32 * hq + h);  // four consecutive k of one core-matrix row
        *reinterpret_cast<float4*>(sm.Ahi + at) = hi;
        *reinterpret_cast<float4*>(sm.Alo + at) = lo;
    }
    // the tile's operands, written by every thread, become visible to the tensor core
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
        tc_fence_after();
        const unsigned ahi = tc_smem(sm.Ahi), alo = tc_smem(sm.Alo), bw = tc_smem(sm.W2f);
        for (int k = 0; k < H / 8; ++k) {
            const unsigned off = (unsigned)k * 2u * TC_LBO;  // K slice k: core matrices 2k, 2k+1
            tc_mma(tmem, tc_desc(ahi + off), tc_desc(bw + off), k > 0);
            tc_mma(tmem, tc_desc(alo + off), tc_desc(bw + off), true);
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                         tc_smem(&sm.bar))
                     : "memory");
    }
    bool done = false;
    for (long it = 0; it < kTcSpin && !done; ++it) done = tc_try_wait(&sm.bar, 0);
    if (__syncthreads_or(done ? 0 : 1)) {
        if (tid == 0) atomicExch(err, 1);
    } else {
        tc_fence_after();
        float v[32], y = 0.f;
        tc_ld32(lane_addr, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            const float z2 = v[q] + sm.b2[32 * hq + q];
            y = fmaf(sm.w3[32 * hq + q], z2 * sigm(z2), y);
        }
        sm.Ahi[hq * TC_M + smp] = y;  // the product is complete: its operands are free
        tc_fence_before();
        __syncthreads();
        if (hq == 0 && valid)
            a.Y[s0 + smp] = b3 + ((sm.Ahi[smp] + sm.Ahi[TC_M + smp]) + (sm.Ahi[2 * TC_M + smp] + sm.Ahi[3 * TC_M + smp]));
    }
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(H) : "memory");
    }
}

mra_status mfail(mra_status s, const std::string& msg) {
    mra::set_last_error(msg.c_str());
    return s;
}

#define MCU(call)                                                                                 \
    do {                                                                                          \
        cudaError_t e_ = (call);                                                                  \
        if (e_ != cudaSuccess)                                                                    \
            return mfail(e_ == cudaErrorMemoryAllocation ? MRA_ERR_OOM : MRA_ERR_CUDA,            \
                         std::string(#call ": ") + cudaGetErrorString(e_));                       \
    } while (0)

}  // namespace

struct mra_mlp {
    int D = 0;
    Layout lay{1};
    int sms = 0;
    int t = 0;  // Adam steps taken
    long N = 0, Nq_cap = 0;
    cudaStream_t stream = nullptr, copy = nullptr;  // copy: input copies beside the kernels
    cudaEvent_t copied = nullptr;
    float *master = nullptr, *m = nullptr, *v = nullptr;
    __nv_bfloat16 *W1b = nullptr, *W2b = nullptr, *w3b = nullptr;
    float *X = nullptr, *T = nullptr, *partial = nullptr, *grad = nullptr, *loss = nullptr;
    float *Xq = nullptr, *Yq = nullptr, *Gq = nullptr;
    int grid_train = 1;
    int* tc_err = nullptr;  // bounded-wait status of the tensor-core forward pass
};

namespace {

MlpArgs args_of(const mra_mlp* n, long N, const float* X) {
    MlpArgs a{};
    a.D = n->D;
    a.N = N;
    a.W1 = n->lay.W1; a.b1 = n->lay.b1; a.W2 = n->lay.W2; a.b2 = n->lay.b2;
    a.w3 = n->lay.w3; a.b3 = n->lay.b3; a.P = n->lay.P;
    a.master = n->master;
    a.W1b = n->W1b; a.W2b = n->W2b; a.w3b = n->w3b;
    a.X = X;
    a.T = n->T;
    a.partial = n->partial;
    return a;
}

// A launch that may start while the stream's previous kernel ends: the kernel itself
// waits for it (griddepcontrol.wait) before it touches what that kernel writes.
template <typename... P, typename... A>
cudaError_t launch_serial(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, P(args)...);
}

mra_status launch_train_pass(mra_mlp* n) {
    if (n->N <= 0) return mfail(MRA_ERR_STATE, "mra_mlp: no training data (mra_mlp_set_data)");
    MlpArgs a = args_of(n, n->N, n->X);
    long ntiles = (n->N + S - 1) / S;
    n->grid_train = (int)std::min<long>(ntiles, n->sms);
    MCU(launch_serial(k_mlp_train, dim3(4 * n->grid_train), dim3(NT), sizeof(TrainSmem), n->stream, a));
    MCU(cudaGetLastError());
    return MRA_OK;
}

mra_status launch_reduce(mra_mlp* n, float* grad_out, float* loss_out, float lr) {
    const Layout& L = n->lay;
    float bc1 = 1.f, bc2 = 1.f;
    if (!grad_out) {
        n->t += 1;
        bc1 = 1.f - std::pow(0.9f, (float)n->t);
        bc2 = 1.f - std::pow(0.999f, (float)n->t);
    }
    long blocks = (L.P + 1 + 255) / 256;
    MCU(launch_serial(k_mlp_reduce_adam, dim3((unsigned)blocks), dim3(256), 0, n->stream, L.P, n->grid_train,
                      (const float*)n->partial, grad_out, loss_out, n->master, n->m, n->v, n->W1b, n->W2b, n->w3b, L.W2,
                      L.b2, L.w3, L.b3, L.b1, lr, bc1, bc2));
    MCU(cudaGetLastError());
    return MRA_OK;
}

mra_status sync_bf16(mra_mlp* n) {
    const Layout& L = n->lay;
    k_mlp_sync_bf16<<<(unsigned)((L.P + 255) / 256), 256, 0, n->stream>>>(L.P, n->master, n->W1b, n->W2b, n->w3b,
                                                                           L.W2, L.b2, L.w3, L.b3, L.b1);
    MCU(cudaGetLastError());
    return MRA_OK;
}

// Queues a prediction's copies and kernels.
mra_status enqueue_predict(mra_mlp* n, const float* x, long N, float* y, float* dydx, int* tc_err) {
    MlpArgs a = args_of(n, N, n->Xq);
    a.Y = n->Yq;
    a.G = n->Gq;
    if (dydx) {
        MCU(cudaMemcpyAsync(n->Xq, x, (size_t)N * n->D * sizeof(float), cudaMemcpyHostToDevice, n->stream));
        // few samples: small tiles over many CTAs (the pass is latency); many: more work per weight load
        if (N <= (long)SQ * 2 * n->sms) {
            const int grid = (int)((N + SQ - 1) / SQ);
            k_mlp_pass<SQ><<<grid, NT, smem_bytes(n->D, SQ), n->stream>>>(a);
        } else {
            const int grid = (int)std::min<long>((N + S - 1) / S, (long)n->sms);
            k_mlp_pass<S><<<grid, NT, smem_bytes(n->D, S), n->stream>>>(a);
        }
    } else {
        // values only: the 128 x 128 layer on the tensor cores (tcgen05), 128 samples per tile
        MCU(cudaMemsetAsync(n->tc_err, 0, sizeof(int), n->stream));
        // The inputs are copied in runs of one tile per SM on a stream of their own, each run's kernel after its
        // copy: the copies (some 260 us for 65,536 samples of 19 from pageable memory) hide all kernels but the last.
        const long run = (long)TC_M * n->sms;
        for (long i0 = 0; i0 < N; i0 += run) {
            const long k = std::min(run, N - i0);
            cudaStream_t cs = N > run ? n->copy : n->stream;
            MCU(cudaMemcpyAsync(n->Xq + i0 * n->D, x + i0 * n->D, (size_t)k * n->D * sizeof(float),
                                cudaMemcpyHostToDevice, cs));
            if (N > run) {
                MCU(cudaEventRecord(n->copied, n->copy));
                MCU(cudaStreamWaitEvent(n->stream, n->copied, 0));
            }
            a.N = k;
            a.X = n->Xq + i0 * n->D;
            a.Y = n->Yq + i0;
            k_mlp_forward_tc<<<(int)((k + TC_M - 1) / TC_M), TC_T, sizeof(TcSmem), n->stream>>>(a, n->tc_err);
        }
    }
    MCU(cudaGetLastError());
    MCU(cudaMemcpyAsync(y, n->Yq, (size_t)N * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    if (dydx) MCU(cudaMemcpyAsync(dydx, n->Gq, (size_t)N * n->D * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    if (!dydx) MCU(cudaMemcpyAsync(tc_err, n->tc_err, sizeof(int), cudaMemcpyDeviceToHost, n->stream));
    return MRA_OK;
}

}  // namespace

extern "C" {

mra_status mra_mlp_create(int32_t n_in, int32_t hidden, uint64_t seed, mra_mlp** out) {
    if (!out) return mfail(MRA_ERR_ARG, "mra_mlp_create: out is NULL");
    *out = nullptr;
    if (n_in < 1 || n_in > MAXD) return mfail(MRA_ERR_ARG, "mra_mlp_create: n_in must be in 1..64");
    if (hidden != H) return mfail(MRA_ERR_ARG, "mra_mlp_create: hidden width must be 128");
    int dev = 0, count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) return mfail(MRA_ERR_NO_DEVICE, "no CUDA device");
    MCU(cudaGetDevice(&dev));
    int major = 0, sms = 0;
    MCU(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    MCU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (major != 10) return mfail(MRA_ERR_NO_DEVICE, "mra_mlp: needs an sm_100 device");
    mra_mlp* n = new mra_mlp();
    n->D = n_in;
    n->lay = Layout(n_in);
    n->sms = sms;
    const long P = n->lay.P;
    auto fail_free = [&](mra_status s) {
        mra_mlp_destroy(n);
        return s;
    };
#define MALLOC(ptr, bytes)                                                                          \
    do {                                                                                            \
        cudaError_t e_ = cudaMalloc((void**)&(ptr), (bytes));                                       \
        if (e_ != cudaSuccess) return fail_free(mfail(MRA_ERR_OOM, "mra_mlp: device allocation"));  \
    } while (0)
    if (cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&n->copy, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&n->copied, cudaEventDisableTiming) != cudaSuccess)
        return fail_free(mfail(MRA_ERR_CUDA, "mra_mlp: stream"));
    MALLOC(n->master, P * sizeof(float));
    MALLOC(n->m, P * sizeof(float));
    MALLOC(n->v, P * sizeof(float));
    MALLOC(n->W1b, (size_t)H * n_in * sizeof(__nv_bfloat16));
    MALLOC(n->W2b, (size_t)H * H * sizeof(__nv_bfloat16));
    MALLOC(n->w3b, (size_t)H * sizeof(__nv_bfloat16));
    MALLOC(n->partial, (size_t)n->sms * (P + 1) * sizeof(float));
    MALLOC(n->grad, (size_t)(P + 1) * sizeof(float));
    MALLOC(n->loss, sizeof(float));
#undef MALLOC
    {
        cudaError_t e = cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(TrainSmem));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_mlp_pass<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(n_in, S));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_mlp_pass<SQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem_bytes(n_in, SQ));
        if (e != cudaSuccess) return fail_free(mfail(MRA_ERR_CUDA, std::string("mra_mlp: smem attribute: ") + cudaGetErrorString(e)));
    }
    {
        cudaError_t e = cudaFuncSetAttribute(k_mlp_forward_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(TcSmem));
        if (e != cudaSuccess) return fail_free(mfail(MRA_ERR_CUDA, std::string("mra_mlp: smem attribute: ") + cudaGetErrorString(e)));
    }
    // Glorot-uniform weights from a host generator, zero biases
    std::vector<float> p(P, 0.f);
    std::mt19937_64 gen(seed);
    auto fill = [&](long off, long count, int fan_in, int fan_out) {
        float lim = std::sqrt(6.f / (float)(fan_in + fan_out));
        std::uniform_real_distribution<float> u(-lim, lim);
        for (long k = 0; k < count; ++k) p[off + k] = u(gen);
    };
    fill(n->lay.W1, (long)H * n_in, n_in, H);
    fill(n->lay.W2, (long)H * H, H, H);
    fill(n->lay.w3, H, H, 1);
    mra_status s = mra_mlp_set_params(n, p.data());
    if (s != MRA_OK) return fail_free(s);
    *out = n;
    return MRA_OK;
}

mra_status mra_mlp_destroy(mra_mlp* n) {
    if (!n) return MRA_OK;
    float* fbufs[] = {n->master, n->m, n->v, n->X, n->T, n->partial, n->grad, n->loss, n->Xq, n->Yq, n->Gq};
    for (float* b : fbufs)
        if (b) cudaFree(b);
    if (n->W1b) cudaFree(n->W1b);
    if (n->W2b) cudaFree(n->W2b);
    if (n->w3b) cudaFree(n->w3b);
    if (n->tc_err) cudaFree(n->tc_err);
    if (n->copied) cudaEventDestroy(n->copied);
    if (n->copy) cudaStreamDestroy(n->copy);
    if (n->stream) cudaStreamDestroy(n->stream);
    delete n;
    return MRA_OK;
}

mra_status mra_mlp_num_params(const mra_mlp* n, int64_t* out) {
    if (!n || !out) return mfail(MRA_ERR_ARG, "mra_mlp_num_params: NULL argument");
    *out = n->lay.P;
    return MRA_OK;
}

mra_status mra_mlp_get_params(mra_mlp* n, float* params) {
    if (!n || !params) return mfail(MRA_ERR_ARG, "mra_mlp_get_params: NULL argument");
    MCU(cudaMemcpyAsync(params, n->master, n->lay.P * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    MCU(cudaStreamSynchronize(n->stream));
    return MRA_OK;
}

mra_status mra_mlp_set_params(mra_mlp* n, const float* params) {
    if (!n || !params) return mfail(MRA_ERR_ARG, "mra_mlp_set_params: NULL argument");
    for (long k = 0; k < n->lay.P; ++k)
        if (!std::isfinite(params[k])) return mfail(MRA_ERR_ARG, "mra_mlp_set_params: non-finite parameter");
    const size_t bytes = n->lay.P * sizeof(float);
    MCU(cudaMemcpyAsync(n->master, params, bytes, cudaMemcpyHostToDevice, n->stream));
    MCU(cudaMemsetAsync(n->m, 0, bytes, n->stream));
    MCU(cudaMemsetAsync(n->v, 0, bytes, n->stream));
    n->t = 0;
    mra_status s = sync_bf16(n);
    if (s != MRA_OK) return s;
    MCU(cudaStreamSynchronize(n->stream));
    return MRA_OK;
}

mra_status mra_mlp_set_data(mra_mlp* n, const float* x, const float* t, int64_t N) {
    if (!n || !x || !t) return mfail(MRA_ERR_ARG, "mra_mlp_set_data: NULL argument");
    if (N < 1 || N > MAXN) return mfail(MRA_ERR_ARG, "mra_mlp_set_data: need 1 <= n <= 65536");
    for (long k = 0; k < N * n->D; ++k)
        if (!std::isfinite(x[k])) return mfail(MRA_ERR_ARG, "mra_mlp_set_data: non-finite input");
    for (long k = 0; k < N; ++k)
        if (!std::isfinite(t[k])) return mfail(MRA_ERR_ARG, "mra_mlp_set_data: non-finite target");
    if (!n->X) {
        MCU(cudaMalloc((void**)&n->X, (size_t)MAXN * n->D * sizeof(float)));
        MCU(cudaMalloc((void**)&n->T, (size_t)MAXN * sizeof(float)));
    }
    MCU(cudaMemcpyAsync(n->X, x, (size_t)N * n->D * sizeof(float), cudaMemcpyHostToDevice, n->stream));
    MCU(cudaMemcpyAsync(n->T, t, (size_t)N * sizeof(float), cudaMemcpyHostToDevice, n->stream));
    n->N = N;
    MCU(cudaStreamSynchronize(n->stream));
    return MRA_OK;
}

mra_status mra_mlp_grad(mra_mlp* n, float* grad, float* loss) {
    if (!n || !grad) return mfail(MRA_ERR_ARG, "mra_mlp_grad: NULL argument");
    mra_status s = launch_train_pass(n);
    if (s != MRA_OK) return s;
    s = launch_reduce(n, n->grad, n->loss, 0.f);
    if (s != MRA_OK) return s;
    MCU(cudaMemcpyAsync(grad, n->grad, n->lay.P * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    float l = 0.f;
    MCU(cudaMemcpyAsync(&l, n->loss, sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    MCU(cudaStreamSynchronize(n->stream));
    if (loss) *loss = l / (float)n->N;
    return MRA_OK;
}

mra_status mra_mlp_train(mra_mlp* n, int32_t steps, float lr, float* loss_out) {
    if (!n) return mfail(MRA_ERR_ARG, "mra_mlp_train: NULL argument");
    if (steps < 0 || !(lr > 0.f) || !std::isfinite(lr)) return mfail(MRA_ERR_ARG, "mra_mlp_train: bad steps or lr");
    for (int k = 0; k < steps; ++k) {
        mra_status s = launch_train_pass(n);
        if (s != MRA_OK) return s;
        s = launch_reduce(n, nullptr, n->loss, lr);
        if (s != MRA_OK) return s;
    }
    float l = 0.f;
    MCU(cudaMemcpyAsync(&l, n->loss, sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    MCU(cudaStreamSynchronize(n->stream));
    if (loss_out) *loss_out = n->N ? l / (float)n->N : 0.f;
    return MRA_OK;
}

mra_status mra_mlp_predict(mra_mlp* n, const float* x, int64_t N, float* y, float* dydx) {
    if (!n || !x || !y) return mfail(MRA_ERR_ARG, "mra_mlp_predict: NULL argument");
    if (N < 1 || N > MAXN) return mfail(MRA_ERR_ARG, "mra_mlp_predict: need 1 <= n <= 65536");
    if (!n->Xq) {
        MCU(cudaMalloc((void**)&n->Xq, (size_t)MAXN * n->D * sizeof(float)));
        MCU(cudaMalloc((void**)&n->Yq, (size_t)MAXN * sizeof(float)));
        MCU(cudaMalloc((void**)&n->Gq, (size_t)MAXN * n->D * sizeof(float)));
    }
    if (!n->tc_err) MCU(cudaMalloc((void**)&n->tc_err, sizeof(int)));
    int tc_err = 0;
    const mra_status s = enqueue_predict(n, x, N, y, dydx, &tc_err);
    if (s != MRA_OK) {  // what was queued on either stream still uses the caller's arrays
        cudaStreamSynchronize(n->copy);
        cudaStreamSynchronize(n->stream);
        return s;
    }
    MCU(cudaStreamSynchronize(n->stream));
    if (tc_err) return mfail(MRA_ERR_TIMEOUT, "mra_mlp_predict: the tensor-core product did not complete in time");
    return MRA_OK;
}

}  // extern "C"
