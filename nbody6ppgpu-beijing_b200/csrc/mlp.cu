// mlp.cu -- training and inference of the learned neighbour-radius model
// (the network and its features are defined in mlp.cuh).
//
// Training is supervised regression on samples logged from plain
// Ahmad-Cohen runs: features of a particle at one regular step and the
// target dlog = log(RS*/RS), where RS* is the radius that would have given
// NNBOPT neighbours at its next regular step (estimated from the count that
// step found, nnb ~ RS^3).  Loss: mean squared error in standardised units.
//
//   mlp_grad_kernel   eight samples per CTA and round, one warp each:
//                     bf16-weight forward pass, FP32 backward pass to the
//                     layers' inputs; then every thread sums its own
//                     parameters' gradients over the samples, in a fixed
//                     order;
//   mlp_reduce        CTA partials summed in block order (deterministic), and
//                     in training the Adam step on the FP32 master copy and
//                     the bf16 copy that every forward pass reads;
//   mlp_steps         both for all the steps of an epoch in one launch.
//
// The model is small (4,609 parameters, ~4.5 kFLOP per sample), so the
// passes run on the FP32 pipes: a batch of 1024 samples is ~10 MFLOP, far
// below what tensor-core tiling would pay for.
#include "nb6_common.cuh"
#include "mlp.cuh"

#include <algorithm>
#include <random>
#include <vector>

namespace {

// Gradient kernel: GW sample streams per block of samples, a CTA each, GK
// samples of a stream per round, a warp each.
constexpr int GW = 4, GK = 8, GS = GW * GK, GRAD_NT = GK * 32;
constexpr int W2S = MLP_H + 8;  // row stride of W2 in shared memory (bf16): 16-byte reads of 8 lanes miss no bank
constexpr int MLP_NSMALL = MLP_NPARAM - MLP_H * MLP_H;   // W1, B1, B2, W3, B3 back to back
// The bf16 copy: the flat parameters, then W2 transposed ([r][k]).
constexpr int W16_T = MLP_SMEM_BYTES / 2;
// What one sample hands from its warp to the gradient sums.
struct MlpSample {
    float h1[MLP_H], dz1[MLP_H], h2[MLP_H], dz2[MLP_H];
    float xn[MLP_IN], d, err2, pad;
};
static_assert(sizeof(MlpSample) % 16 == 0, "float4 reads of the sample rows");

// What the CTAs of mlp_steps wait on, each word in a line of its own, and what
// a training run reports.
struct TrainSync {
    unsigned done_grad, pad0[31], done_red, pad1[31];
    float loss;
    unsigned err;   // a wait ran out
};

struct MlpState {
    bool have = false;      // parameters set or trained
    int enabled = 0;        // proposals in regular-force calls
    std::vector<float> host;  // FP32 parameters + moments
    DevBuf<float> w32, m1, m2, grad, part, norm, dx, dy;
    DevBuf<__nv_bfloat16> w16;
    DevBuf<int> perm;          // one epoch's order, then its bias corrections (float2 per step)
    DevBuf<double> mom;
    DevBuf<TrainSync> sync;
    long long adam_t = 0;
};
MlpState M;

// Parameter k into the bf16 copies.
NB6_DEV void store_bf16(__nv_bfloat16 *w16, int k, float w) {
    const __nv_bfloat16 v = __float2bfloat16_rn(w);
    w16[k] = v;
    const int q = k - MLP_OFF_W2;
    if (q >= 0 && q < MLP_H * MLP_H) w16[W16_T + (q % MLP_H) * MLP_H + q / MLP_H] = v;
}

__global__ void mlp_to_bf16(const float *__restrict__ w32, __nv_bfloat16 *__restrict__ w16) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < MLP_SMEM_BYTES / 2; k += gridDim.x * blockDim.x)
        store_bf16(w16, k, k < MLP_NPARAM ? w32[k] : 0.0f);
}

// The kernels of a gradient, and of training steps too large for mlp_steps, are
// launched back to back, each allowed on the SMs while the one before drains (programmatic dependent launch): it
// waits here before it touches what that one wrote.
NB6_DEV void wait_for_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
NB6_DEV void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Eight bf16 weights (one 16-byte read) times eight inputs, in index order.
NB6_DEV float fma8(const __nv_bfloat16 *w, const float *in, float z) {
    const uint4 p = *reinterpret_cast<const uint4 *>(w);
    const float4 a = *reinterpret_cast<const float4 *>(in), b = *reinterpret_cast<const float4 *>(in + 4);
    const unsigned q[4] = {p.x, p.y, p.z, p.w};
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        z = fmaf(__uint_as_float(q[c] << 16), v[2 * c], z);
        z = fmaf(__uint_as_float(q[c] & 0xffff0000u), v[2 * c + 1], z);
    }
    return z;
}

// Gradient of sum_s (out_s - y_s)^2 / n over the samples [off, off + cnt)
// of the (optionally permuted) set; per-CTA partials into part[block][.],
// squared-error partials into part_loss[block].
//
// Sample q = (block GW + w) + k (blocks GW) is the k-th of stream w of its
// block.  A parameter's gradient is summed over k within a stream, then over
// the streams, then over the blocks, so the sums do not depend on how many
// samples run at a time.  Eight samples of a stream are in flight (a warp
// each), the four streams of a block on different SMs: with one warp per stream
// the kernel was a chain of eight samples' forward and backward passes and of
// 8,192 read-modify-writes each of a gradient buffer in shared memory (45 us
// for 1,024 samples); with the block's 32 warps in one CTA the shared-memory
// reads of 32 SMs bounded it (16 us, now 11).  The layers read eight weights per
// 16-byte load, W2 along its rows (backward) and, from the transposed copy,
// along its columns (forward).
struct GradSmem {
    __align__(16) __nv_bfloat16 sw[(MLP_NSMALL + 7) / 8 * 8];   // W1, B1 | B2, W3, B3
    __align__(16) __nv_bfloat16 w2[MLP_H * W2S], w2t[MLP_H * W2S];
    __align__(16) MlpSample smp[GK];
};
struct GradArgs {
    int cnt;        // samples of the batch
    float inv_n;
    const float *x, *y;
    const int *perm;
    const __nv_bfloat16 *w16;
    const float *norm;
    float *part, *part_loss;
};
// A warp's sample of a round: its standardised inputs and target.
struct SampleIn {
    float xn[MLP_IN], target;
    bool have;
};
// The sample of stream `first` at `base` samples into the batch at `off`.
NB6_DEV void fetch_sample(const GradArgs &g, int off, int base, int first, int stride, SampleIn &in) {
    const int q = base + (int)(threadIdx.x >> 5) * stride + first;
    in.have = q < g.cnt;
    if (!in.have) return;
    const int s = g.perm ? g.perm[off + q] : off + q;
#pragma unroll
    for (int k = 0; k < MLP_IN; ++k) in.xn[k] = (g.x[(size_t)s * MLP_IN + k] - g.norm[k]) * g.norm[MLP_IN + k];
    in.target = g.y[s];
}

// The gradient sums of stream `first`, whose first sample is in `in`.
NB6_DEV void grad_pass(GradSmem &sm, const GradArgs &g, int off, int first, int stride, SampleIn &in) {
    constexpr int B2 = MLP_OFF_W2, W3 = B2 + MLP_H, B3 = W3 + MLP_H;   // places in sw
    const __nv_bfloat16 *sw = sm.sw, *w2 = sm.w2, *w2t = sm.w2t;
    MlpSample *smp = sm.smp;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cnt = g.cnt;
    const float inv_n = g.inv_n, ymean = g.norm[2 * MLP_IN], yinv = 1.0f / g.norm[2 * MLP_IN + 1];
    const float (&xn)[MLP_IN] = in.xn;
    const uint4 *src = reinterpret_cast<const uint4 *>(g.w16);
    for (int q = tid; q < MLP_H * MLP_H / 8; q += GRAD_NT) {
        const int r = q / (MLP_H / 8), c = q % (MLP_H / 8);
        reinterpret_cast<uint4 *>(sm.w2 + r * W2S)[c] = __ldcg(src + MLP_OFF_W2 / 8 + q);
        reinterpret_cast<uint4 *>(sm.w2t + r * W2S)[c] = __ldcg(src + W16_T / 8 + q);
    }
    for (int q = tid; q < (MLP_NSMALL + 7) / 8; q += GRAD_NT)
        reinterpret_cast<uint4 *>(sm.sw)[q] = __ldcg(src + (q < MLP_OFF_W2 / 8 ? q : q + MLP_H * MLP_H / 8));
    __syncthreads();
    // this thread's parameters: W2[gk][gr .. gr+15], and others
    const int gk = tid >> 2, gr = (tid & 3) * 16;
    constexpr int NO = (MLP_NSMALL + GRAD_NT - 1) / GRAD_NT;
    float g2[16], g1[NO], lsum = 0.0f;
#pragma unroll
    for (int c = 0; c < 16; ++c) g2[c] = 0.0f;
#pragma unroll
    for (int c = 0; c < NO; ++c) g1[c] = 0.0f;
    MlpSample &S = smp[warp];
    for (int base = 0; base < cnt; base += GK * stride) {
        // forward and backward pass of this warp's sample
        if (in.have) {
            float z1[2], z2[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int r = lane + 32 * u;
                float z = bf(sw, MLP_OFF_B1 + r);
#pragma unroll
                for (int k = 0; k < MLP_IN; ++k) z = fmaf(bf(sw, MLP_OFF_W1 + k * MLP_H + r), xn[k], z);
                z1[u] = z;
                S.h1[r] = mlp_silu(z);
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 2; ++u) z2[u] = bf(sw, B2 + lane + 32 * u);
#pragma unroll
            for (int k = 0; k < MLP_H; k += 8)
#pragma unroll
                for (int u = 0; u < 2; ++u) z2[u] = fma8(w2t + (lane + 32 * u) * W2S + k, S.h1 + k, z2[u]);
            const float h2[2] = {mlp_silu(z2[0]), mlp_silu(z2[1])};
            float o = bf(sw, W3 + lane) * h2[0] + bf(sw, W3 + lane + 32) * h2[1];
#pragma unroll
            for (int t = 16; t > 0; t >>= 1) o += __shfl_xor_sync(0xffffffffu, o, t);
            const float out = o + bf(sw, B3);
            const float err = out - (in.target - ymean) * yinv;
            const float d = 2.0f * err * inv_n;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int r = lane + 32 * u;
                S.h2[r] = h2[u];
                S.dz2[r] = d * bf(sw, W3 + r) * mlp_dsilu(z2[u]);
            }
            __syncwarp();
            float dh1[2] = {0.0f, 0.0f};
#pragma unroll
            for (int k = 0; k < MLP_H; k += 8)
#pragma unroll
                for (int u = 0; u < 2; ++u) dh1[u] = fma8(w2 + (lane + 32 * u) * W2S + k, S.dz2 + k, dh1[u]);
#pragma unroll
            for (int u = 0; u < 2; ++u) S.dz1[lane + 32 * u] = dh1[u] * mlp_dsilu(z1[u]);
            if (lane == 0) {
#pragma unroll
                for (int k = 0; k < MLP_IN; ++k) S.xn[k] = xn[k];
                S.d = d;
                S.err2 = err;
            }
        } else {   // no sample: every product below is zero
            for (int k = lane; k < (int)(sizeof(MlpSample) / 4); k += 32) reinterpret_cast<float *>(&S)[k] = 0.0f;
        }
        fetch_sample(g, off, base + GK * stride, first, stride, in);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < GK; ++k) {
            const MlpSample &T = smp[k];
            const float h = T.h1[gk];
#pragma unroll
            for (int c = 0; c < 16; c += 4) {
                const float4 z = *reinterpret_cast<const float4 *>(&T.dz2[gr + c]);
                g2[c] = fmaf(z.x, h, g2[c]);
                g2[c + 1] = fmaf(z.y, h, g2[c + 1]);
                g2[c + 2] = fmaf(z.z, h, g2[c + 2]);
                g2[c + 3] = fmaf(z.w, h, g2[c + 3]);
            }
        }
        // the other parameters: W1, B1, B2, W3, B3 and the loss
#pragma unroll
        for (int c = 0; c < NO; ++c) {
            const int p = tid + c * GRAD_NT, r = p % MLP_H;
#pragma unroll
            for (int k = 0; k < GK; ++k) {
                const MlpSample &T = smp[k];
                if (p < MLP_OFF_B1) g1[c] = fmaf(T.dz1[r], T.xn[p / MLP_H], g1[c]);
                else if (p < B2) g1[c] += T.dz1[r];
                else if (p < W3) g1[c] += T.dz2[r];
                else if (p < B3) g1[c] = fmaf(T.d, T.h2[r], g1[c]);
                else if (p == B3) {
                    g1[c] += T.d;
                    lsum = fmaf(T.err2, T.err2, lsum);
                }
            }
        }
        __syncthreads();
    }
    float *o = g.part + (size_t)first * MLP_NPARAM;
#pragma unroll
    for (int c = 0; c < 16; ++c) o[MLP_OFF_W2 + gk * MLP_H + gr + c] = g2[c];
#pragma unroll
    for (int c = 0; c < NO; ++c) {
        const int p = tid + c * GRAD_NT;
        if (p < MLP_NSMALL) o[p < MLP_OFF_W2 ? p : p + MLP_H * MLP_H] = g1[c];
        if (p == B3) g.part_loss[first] = lsum;
    }
}

__global__ void __launch_bounds__(GRAD_NT) mlp_grad_kernel(const GradArgs g, int off) {
    __shared__ GradSmem sm;
    let_next_start();
    const int stride = gridDim.x * GW, first = blockIdx.x * GW + blockIdx.y;
    SampleIn in;
    fetch_sample(g, off, 0, first, stride, in);
    wait_for_previous();   // the weights
    grad_pass(sm, g, off, first, stride, in);
}

// The Adam step of one training batch.
struct AdamArgs {
    float *w, *m1, *m2;
    __nv_bfloat16 *w16;
    float lr, b1, b2, eps, bc1, bc2;
};

// grad[k] = sum over blocks, in order, of the sum over a block's streams;
// loss[0] += sum of squared errors, likewise (as parameter MLP_NPARAM).  ADAM:
// then the step on parameter k and its bf16 copies, which the next batch's
// forward pass reads, in the same launch.  A CTA takes RED_P parameters; its
// threads sum the streams of 32 blocks side by side (one memory round trip; a
// thread per parameter walked 128 partials, 10 us for a batch of 1,024), then
// one warp adds the blocks in order.
constexpr int RED_P = 32, RED_NT = 256;
static_assert(GW == 4, "mlp_reduce adds four streams");
template <bool ADAM>
NB6_DEV void reduce_slice(int slice, int nb, const float *part, const float *part_loss, float *grad, float *loss,
                          const AdamArgs &ad, float (*acc)[RED_P]) {
    const int p = threadIdx.x % RED_P, row = threadIdx.x / RED_P, k = slice * RED_P + p;
    const float *src = k < MLP_NPARAM ? part + k : part_loss;
    const size_t step = k < MLP_NPARAM ? MLP_NPARAM : 1;
    const bool mine = row == 0 && k < MLP_NPARAM;
    float m1 = 0.f, m2 = 0.f, w = 0.f, g = 0.f;
    if (ADAM && mine) {
        m1 = ad.m1[k];
        m2 = ad.m2[k];
        w = ad.w[k];
    }
    for (int b0 = 0; b0 < nb; b0 += 32) {
#pragma unroll
        for (int r = row; r < 32; r += RED_NT / RED_P) {
            if (b0 + r < nb && k <= MLP_NPARAM) {
                const float *q = src + (size_t)(b0 + r) * GW * step;
                acc[r][p] = ((__ldcg(q) + __ldcg(q + step)) + __ldcg(q + 2 * step)) + __ldcg(q + 3 * step);
            }
        }
        __syncthreads();
        if (row == 0 && k <= MLP_NPARAM) {
            const int n = min(32, nb - b0);
#pragma unroll 8
            for (int r = 0; r < n; ++r) g += acc[r][p];
        }
        __syncthreads();
    }
    if (mine) {
        if (ADAM) {
            const float a = ad.b1 * m1 + (1.0f - ad.b1) * g;
            const float b = ad.b2 * m2 + (1.0f - ad.b2) * g * g;
            ad.m1[k] = a;
            ad.m2[k] = b;
            w -= ad.lr * (a / ad.bc1) / (sqrtf(b / ad.bc2) + ad.eps);
            ad.w[k] = w;
            store_bf16(ad.w16, k, w);
        } else {
            grad[k] = g;
        }
    } else if (row == 0 && k == MLP_NPARAM) {
        loss[0] += g;
    }
}

template <bool ADAM>
__global__ void __launch_bounds__(RED_NT)
    mlp_reduce(int nb, const float *part, const float *part_loss, float *grad, float *loss, const AdamArgs ad) {
    __shared__ float acc[32][RED_P];
    let_next_start();
    wait_for_previous();
    reduce_slice<ADAM>(blockIdx.x, nb, part, part_loss, grad, loss, ad, acc);
}

// Wait until *count has reached `target`; false (and *err set) after WAIT_MAX
// polls, about a second.
constexpr int WAIT_MAX = 1 << 21;
NB6_DEV bool wait_count(const unsigned *count, unsigned target, unsigned *err) {
    int bad = 0;
    if (threadIdx.x == 0) {
        bad = 1;
        for (int t = 0; t < WAIT_MAX && bad; ++t) {
            unsigned c;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
            bad = (int)(c - target) < 0;
        }
        if (bad) *err = 1u;
    }
    return !__syncthreads_or(bad);
}
NB6_DEV void add_count(unsigned *count) {
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
}

// A run of training steps in one cooperative launch: CTA c < ngrad is stream
// c of a batch, CTA c < nred sums and steps slices of the parameters, and two
// counters in global memory (partials written, parameters written) order the
// phases.  Same sums in the same order as mlp_grad_kernel and mlp_reduce.  A
// step is a chain of short phases, so what a launch costs (its start, the
// drain before it) was a third of it: 32 steps of 1,024 samples 845 us as 64
// launches, with the upload and the host's shuffle (some 350 us), now 670.  The
// next batch's samples are fetched before the wait for the parameters.
constexpr int NSLICE = MLP_NPARAM / RED_P + 1;   // every parameter, and the loss
__global__ void __launch_bounds__(GRAD_NT)
    mlp_steps(const GradArgs g, int nb, int step0, int steps, const float2 *__restrict__ bc, AdamArgs ad,
              TrainSync *sync) {
    __shared__ GradSmem sm;
    __shared__ float acc[32][RED_P];
    const int stride = nb * GW, first = blockIdx.x, nred = min((int)gridDim.x, NSLICE);
    const bool grads = first < stride;
    SampleIn in;
    if (grads) fetch_sample(g, step0 * g.cnt, 0, first, stride, in);
    for (int s = step0; s < step0 + steps; ++s) {
        if (grads) {
            grad_pass(sm, g, s * g.cnt, first, stride, in);
            add_count(&sync->done_grad);
            if (s + 1 < step0 + steps) fetch_sample(g, (s + 1) * g.cnt, 0, first, stride, in);
        }
        if (first < nred) {
            if (!wait_count(&sync->done_grad, (unsigned)(s + 1) * stride, &sync->err)) return;
            const float2 b = bc[s];
            ad.bc1 = b.x;
            ad.bc2 = b.y;
            for (int k = first; k < NSLICE; k += nred)
                reduce_slice<true>(k, nb, g.part, g.part_loss, nullptr, &sync->loss, ad, acc);
            add_count(&sync->done_red);
        }
        if (grads && s + 1 < step0 + steps &&
            !wait_count(&sync->done_red, (unsigned)(s + 1) * nred, &sync->err))
            return;
    }
}

__global__ void __launch_bounds__(128)
    mlp_predict_kernel(int n, const float *__restrict__ x, float *__restrict__ y,
                       const __nv_bfloat16 *__restrict__ w16, const float *__restrict__ norm) {
    __shared__ __align__(16) __nv_bfloat16 sw[MLP_SMEM_BYTES / 2];
    mlp_load(sw, w16);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int s = blockIdx.x * 4 + warp; s < n; s += gridDim.x * 4) {
        float f[MLP_IN];
#pragma unroll
        for (int k = 0; k < MLP_IN; ++k) f[k] = x[(size_t)s * MLP_IN + k];
        MlpAct a;
        const float out = mlp_forward_warp(sw, norm, f, lane, a);
        if (lane == 0) y[s] = out * norm[2 * MLP_IN + 1] + norm[2 * MLP_IN];
    }
}

// Moments of the training samples: sums and sums of squares of the five
// inputs and the target in FP64 (per thread, lane tree, warps, then CTAs in
// order: deterministic), and from them the stored moments (mean, 1 / std of
// the inputs, mean, std of the target).  The host's pass over 32,768 samples
// took 0.4 ms of a one-epoch run.
constexpr int MOM_NT = 256, MOM_CTAS = 64, MOM_N = 2 * (MLP_IN + 1);
__global__ void __launch_bounds__(MOM_NT)
    mlp_moment_sums(int n, const float *__restrict__ x, const float *__restrict__ y, double *__restrict__ part) {
    __shared__ double red[MOM_NT / 32][MOM_N];
    double s[MOM_N] = {};
    for (int q = blockIdx.x * MOM_NT + threadIdx.x; q < n; q += gridDim.x * MOM_NT)
#pragma unroll
        for (int k = 0; k <= MLP_IN; ++k) {
            const double v = k < MLP_IN ? x[(size_t)q * MLP_IN + k] : y[q];
            s[2 * k] += v;
            s[2 * k + 1] += v * v;
        }
#pragma unroll
    for (int c = 0; c < MOM_N; ++c) {
        const double w = warp_sum_d(s[c]);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][c] = w;
    }
    __syncthreads();
    if (threadIdx.x < MOM_N) {
        double w = 0.0;
        for (int q = 0; q < MOM_NT / 32; ++q) w += red[q][threadIdx.x];
        part[blockIdx.x * MOM_N + threadIdx.x] = w;
    }
}

__global__ void __launch_bounds__(32) mlp_moments(int n, const double *__restrict__ part, float *__restrict__ norm) {
    const int k = threadIdx.x;
    if (k > MLP_IN) return;
    double s1 = 0.0, s2 = 0.0;
#pragma unroll 8
    for (int b = 0; b < MOM_CTAS; ++b) {
        s1 += part[b * MOM_N + 2 * k];
        s2 += part[b * MOM_N + 2 * k + 1];
    }
    const double mean = s1 / n, v = s2 / n - mean * mean;
    const double var = v < 1e-12 ? 1e-12 : v;   // (a NaN stays one, as the mean does; fmax would drop it)
    if (k < MLP_IN) {
        norm[k] = (float)mean;
        norm[MLP_IN + k] = (float)(1.0 / sqrt(var));
    } else {
        norm[2 * MLP_IN] = (float)mean;
        norm[2 * MLP_IN + 1] = (float)sqrt(var);
    }
}

void mlp_alloc() {
    if (M.w32.ptr) return;
    nb6_devinit_once(0);
    M.w32.reserve(MLP_NPARAM);
    M.m1.reserve(MLP_NPARAM);
    M.m2.reserve(MLP_NPARAM);
    M.grad.reserve(MLP_NPARAM);
    M.norm.reserve(MLP_NNORM);
    M.sync.reserve(1);
    M.mom.reserve(MOM_CTAS * MOM_N);
    M.w16.reserve(W16_T + MLP_H * MLP_H);
    M.host.assign(MLP_NPARAM + MLP_NNORM, 0.0f);
}

// Host copy -> device FP32 master, moments and the bf16 copy; resets Adam.
void mlp_upload() {
    cudaStream_t st = nb6_stream();
    NB6_CUDA_CHECK(cudaMemcpyAsync(M.w32.ptr, M.host.data(), sizeof(float) * MLP_NPARAM,
                                   cudaMemcpyHostToDevice, st));
    NB6_CUDA_CHECK(cudaMemcpyAsync(M.norm.ptr, M.host.data() + MLP_NPARAM, sizeof(float) * MLP_NNORM,
                                   cudaMemcpyHostToDevice, st));
    NB6_CUDA_CHECK(cudaMemsetAsync(M.m1.ptr, 0, sizeof(float) * MLP_NPARAM, st));
    NB6_CUDA_CHECK(cudaMemsetAsync(M.m2.ptr, 0, sizeof(float) * MLP_NPARAM, st));
    mlp_to_bf16<<<(MLP_SMEM_BYTES / 2 + 255) / 256, 256, 0, st>>>(M.w32.ptr, M.w16.ptr);
    NB6_CUDA_CHECK(cudaGetLastError());
    NB6_CUDA_CHECK(cudaStreamSynchronize(st));
    M.adam_t = 0;
    M.have = true;
}

// Parameters and moments -> host copy.
void mlp_download() {
    NB6_CUDA_CHECK(cudaStreamSynchronize(nb6_stream()));
    NB6_CUDA_CHECK(cudaMemcpy(M.host.data(), M.w32.ptr, sizeof(float) * MLP_NPARAM, cudaMemcpyDeviceToHost));
    NB6_CUDA_CHECK(cudaMemcpy(M.host.data() + MLP_NPARAM, M.norm.ptr, sizeof(float) * MLP_NNORM,
                              cudaMemcpyDeviceToHost));
}

void mlp_upload_samples(int n, const float *x, const float *y) {
    cudaStream_t st = nb6_stream();
    M.dx.reserve((size_t)n * MLP_IN);
    const Nb6Seg sx{0, x, sizeof(float) * MLP_IN * (size_t)n};
    nb6_upload(M.dx.ptr, &sx, 1, sx.len, st);
    if (y) {
        M.dy.reserve(n);
        const Nb6Seg sy{0, y, sizeof(float) * (size_t)n};
        nb6_upload(M.dy.ptr, &sy, 1, sy.len, st);
    }
}

int grad_blocks(int cnt) { return std::max(1, std::min((cnt + GS - 1) / GS, nb6_num_sms() * 2)); }

GradArgs grad_args(int cnt, int nb, const int *perm) {
    M.part.reserve((size_t)nb * GW * (MLP_NPARAM + 1));
    return GradArgs{cnt,        1.0f / (float)cnt, M.dx.ptr,   M.dy.ptr,   perm,
                    M.w16.ptr,  M.norm.ptr,        M.part.ptr, M.part.ptr + (size_t)nb * GW * MLP_NPARAM};
}

// One gradient over samples [off, off+cnt) of the uploaded set: into M.grad,
// or through the Adam step `adam` into the parameters.
void mlp_grad_launch(int cnt, int off, const int *perm, const AdamArgs *adam, cudaStream_t st) {
    const int nb = grad_blocks(cnt);
    const GradArgs g = grad_args(cnt, nb, perm);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    c.gridDim = dim3(nb, GW);
    c.blockDim = dim3(GRAD_NT);
    NB6_CUDA_CHECK(cudaLaunchKernelEx(&c, mlp_grad_kernel, g, off));
    c.gridDim = dim3(NSLICE);
    c.blockDim = dim3(RED_NT);
    const AdamArgs ad = adam ? *adam : AdamArgs{};
    NB6_CUDA_CHECK(cudaLaunchKernelEx(&c, adam ? mlp_reduce<true> : mlp_reduce<false>, nb, (const float *)g.part,
                                      (const float *)g.part_loss, M.grad.ptr, &M.sync.ptr->loss, ad));
}

// CTAs of mlp_steps that the device holds at a time; 0 without cooperative
// launches.
int steps_capacity() {
    static const int cap = [] {
        int dev = 0, coop = 0, occ = 0;
        NB6_CUDA_CHECK(cudaGetDevice(&dev));
        NB6_CUDA_CHECK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        NB6_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, mlp_steps, GRAD_NT, 0));
        return coop ? occ * nb6_num_sms() : 0;
    }();
    return cap;
}

// The training steps of one epoch; bc[s] are the bias corrections of step s.
// One launch of mlp_steps per STEPS_MAX of them when a batch's CTAs are all on
// the device at once and its step is short, else two launches a step.
void mlp_train_steps(int B, int steps, const float2 *bc, const float2 *dbc, AdamArgs ad, cudaStream_t st) {
    constexpr int STEPS_MAX = 1024, BATCH_MAX = 1 << 20;   // (a step within a millisecond or so)
    const int nb = grad_blocks(B), ctas = std::max(nb * GW, std::min(NSLICE, nb6_num_sms()));
    if (ctas > steps_capacity() || B > BATCH_MAX) {
        for (int s = 0; s < steps; ++s) {
            ad.bc1 = bc[s].x;
            ad.bc2 = bc[s].y;
            mlp_grad_launch(B, s * B, M.perm.ptr, &ad, st);
        }
        return;
    }
    GradArgs g = grad_args(B, nb, M.perm.ptr);
    TrainSync *sync = M.sync.ptr;
    for (int s0 = 0; s0 < steps; s0 += STEPS_MAX) {
        int n = std::min(STEPS_MAX, steps - s0), b = nb;
        void *arg[] = {&g, &b, &s0, &n, &dbc, &ad, &sync};
        NB6_CUDA_CHECK(
            cudaLaunchCooperativeKernel((const void *)mlp_steps, dim3(ctas), dim3(GRAD_NT), arg, 0, st));
    }
}

bool check_n(int n) {
    if (n <= 0) {
        nb6_fatal(NB6_ERR_BAD_ARG);
        return false;
    }
    return true;
}

}  // namespace

// Epilogue arguments for the regular-force call: proposals on when enabled
// and a model is loaded.
MlpArgs nb6_mlp_args(const double *h2, const double *dtr) {
    MlpArgs a;
    a.h2 = h2;
    a.dtr = dtr;
    a.w = M.w16.ptr;
    a.norm = M.norm.ptr;
    a.on = (M.enabled && M.have) ? 1 : 0;
    return a;
}

extern "C" {

// Number of floats of a model: parameters (see mlp.cuh for the layout)
// followed by the moments in_mean[5], in_scale[5], out_mean, out_std.
int nb6_mlp_size_(void) { return MLP_NPARAM + MLP_NNORM; }

// Random initial parameters (He-scaled normal, zero biases), identity moments.
void nb6_mlp_init_(int *seed) {
    mlp_alloc();
    std::mt19937 gen((unsigned)*seed);
    auto fill = [&](int off, int fan_in, int count) {
        std::normal_distribution<float> d(0.0f, std::sqrt(2.0f / (float)fan_in));
        for (int k = 0; k < count; ++k) M.host[off + k] = d(gen);
    };
    std::fill(M.host.begin(), M.host.end(), 0.0f);
    fill(MLP_OFF_W1, MLP_IN, MLP_IN * MLP_H);
    fill(MLP_OFF_W2, MLP_H, MLP_H * MLP_H);
    fill(MLP_OFF_W3, MLP_H, MLP_H);
    float *nm = M.host.data() + MLP_NPARAM;
    for (int k = 0; k < MLP_IN; ++k) nm[MLP_IN + k] = 1.0f;
    nm[2 * MLP_IN + 1] = 1.0f;
    mlp_upload();
}

void nb6_mlp_set_(const float *model) {
    mlp_alloc();
    std::copy(model, model + MLP_NPARAM + MLP_NNORM, M.host.begin());
    mlp_upload();
}

void nb6_mlp_get_(float *model) {
    if (!M.have) {
        nb6_fatal(NB6_ERR_NOT_OPEN);
        return;
    }
    mlp_download();
    std::copy(M.host.begin(), M.host.end(), model);
}

// Gradient of the mean squared error (standardised units) over n samples
// x[n][5], y[n] at the current parameters, and the loss.  Deterministic.
void nb6_mlp_grad_(int *n, const float *x, const float *y, float *grad, float *loss) {
    if (!M.have) {
        nb6_fatal(NB6_ERR_NOT_OPEN);
        return;
    }
    if (!check_n(*n)) return;
    mlp_upload_samples(*n, x, y);
    cudaStream_t st = nb6_stream();
    NB6_CUDA_CHECK(cudaMemsetAsync(M.sync.ptr, 0, sizeof(TrainSync), st));
    mlp_grad_launch(*n, 0, nullptr, nullptr, st);
    NB6_CUDA_CHECK(cudaStreamSynchronize(st));
    NB6_CUDA_CHECK(cudaMemcpy(grad, M.grad.ptr, sizeof(float) * MLP_NPARAM, cudaMemcpyDeviceToHost));
    float l = 0.0f;
    NB6_CUDA_CHECK(cudaMemcpy(&l, &M.sync.ptr->loss, sizeof(float), cudaMemcpyDeviceToHost));
    *loss = l / (float)*n;
}

// Train on n samples: moments from the data, then `epochs` passes of Adam
// over shuffled mini-batches of `batch`.  loss_hist[e] = mean squared error
// (standardised) over epoch e.  Starts from the current parameters (call
// nb6_mlp_init_ first for a fresh model).
void nb6_mlp_train_(int *n_, const float *x, const float *y, int *epochs, int *batch, float *lr, int *seed,
                    float *loss_hist) {
    const int n = *n_, B = std::max(1, std::min(*batch, n));
    if (!check_n(n) || *epochs < 0) return;
    mlp_alloc();
    if (!M.have) {
        int s = *seed;
        nb6_mlp_init_(&s);
    }
    // the device parameters stay; moments of the inputs and the target, and a
    // fresh optimiser
    cudaStream_t st = nb6_stream();
    mlp_upload_samples(n, x, y);
    mlp_moment_sums<<<MOM_CTAS, MOM_NT, 0, st>>>(n, M.dx.ptr, M.dy.ptr, M.mom.ptr);
    mlp_moments<<<1, 32, 0, st>>>(n, M.mom.ptr, M.norm.ptr);
    NB6_CUDA_CHECK(cudaGetLastError());
    NB6_CUDA_CHECK(cudaMemsetAsync(M.m1.ptr, 0, sizeof(float) * MLP_NPARAM, st));
    NB6_CUDA_CHECK(cudaMemsetAsync(M.m2.ptr, 0, sizeof(float) * MLP_NPARAM, st));
    M.adam_t = 0;
    const int steps = n / B;
    const size_t bc_at = ((size_t)n + 1) / 2 * 2;   // in ints, 8-byte aligned
    M.perm.reserve(bc_at + 2 * (size_t)steps);
    std::vector<int> perm(n);
    std::vector<float2> bc(steps);
    for (int q = 0; q < n; ++q) perm[q] = q;
    std::mt19937 gen((unsigned)*seed);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const AdamArgs ad{M.w32.ptr, M.m1.ptr, M.m2.ptr, M.w16.ptr, *lr, b1, b2, eps, 1.0f, 1.0f};
    if (*epochs > 0) std::shuffle(perm.begin(), perm.end(), gen);
    for (int e = 0; e < *epochs; ++e) {
        for (float2 &c : bc) {
            M.adam_t++;
            c = make_float2(1.0f - std::pow(b1, (float)M.adam_t), 1.0f - std::pow(b2, (float)M.adam_t));
        }
        const Nb6Seg sp[2] = {{0, perm.data(), sizeof(int) * (size_t)n},
                              {sizeof(int) * bc_at, bc.data(), sizeof(float2) * (size_t)steps}};
        nb6_upload(M.perm.ptr, sp, 2, sp[1].off + sp[1].len, st);
        NB6_CUDA_CHECK(cudaMemsetAsync(M.sync.ptr, 0, sizeof(TrainSync), st));
        mlp_train_steps(B, steps, bc.data(), reinterpret_cast<const float2 *>(M.perm.ptr + bc_at), ad, st);
        // (the next epoch's order, while the GPU works on this one's)
        if (e + 1 < *epochs) std::shuffle(perm.begin(), perm.end(), gen);
        NB6_CUDA_CHECK(cudaStreamSynchronize(st));
        struct {
            float loss;
            unsigned err;
        } res{};
        static_assert(offsetof(TrainSync, err) == offsetof(TrainSync, loss) + sizeof(float), "read together");
        NB6_CUDA_CHECK(cudaMemcpy(&res, &M.sync.ptr->loss, sizeof(res), cudaMemcpyDeviceToHost));
        if (res.err) {
            nb6_fatal(NB6_ERR_WAIT_TIMEOUT);
            return;
        }
        if (loss_hist) loss_hist[e] = res.loss / (float)(steps * B);
    }
    mlp_download();
}

// y[n] = model output (dlog RS) for x[n][5], bf16 parameters, FP32 sums.
void nb6_mlp_predict_(int *n, const float *x, float *y) {
    if (!M.have) {
        nb6_fatal(NB6_ERR_NOT_OPEN);
        return;
    }
    if (!check_n(*n)) return;
    mlp_upload_samples(*n, x, nullptr);
    DevBuf<float> out;
    out.reserve(*n);
    cudaStream_t st = nb6_stream();
    const int blocks = std::max(1, std::min((*n + 3) / 4, nb6_num_sms() * 8));
    mlp_predict_kernel<<<blocks, 128, 0, st>>>(*n, M.dx.ptr, out.ptr, M.w16.ptr, M.norm.ptr);
    NB6_CUDA_CHECK(cudaGetLastError());
    NB6_CUDA_CHECK(cudaStreamSynchronize(st));
    NB6_CUDA_CHECK(cudaMemcpy(y, out.ptr, sizeof(float) * (size_t)*n, cudaMemcpyDeviceToHost));
    out.release();
}

// Radius proposals in regular-force calls on (1) or off (0).
void nb6_mlp_enable_(int *flag) {
    if (*flag && !M.have) {
        nb6_fatal(NB6_ERR_NOT_OPEN);
        return;
    }
    M.enabled = *flag ? 1 : 0;
}

}  // extern "C"
