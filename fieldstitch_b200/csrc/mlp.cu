// Learned match filter: an 8-64-64-1 MLP over per-correspondence features, trained on the GPU.
//
// The plain guided matcher (matching._guided, app/planesite/matching.py:113-152) accepts a
// query's best candidate when it passes the ratio test; the pipeline then verifies the accepted
// set geometrically (RANSAC homography, matching.py:205-233). Here the candidates that the plain
// matcher sees (best target, b1, b2 for every query) are described by 8 features and scored by
// a small MLP trained on labels that the plain pipeline's own verification produces; the plain
// ratio test remains the fallback.
//
//   k_mlp_features    features of every query's best candidate:
//                     0 ratio sqrt(b1) / sqrt(b2) (0 for a single candidate), 1 sqrt(b1) / 512,
//                     2 log2(size_b / size_a), 3 signed angle difference / 180 (wrapped),
//                     4 prior residual |pred_a - xy_b| / radius, 5 response_a, 6 response_b,
//                     7 octave_a
//   k_mlp_fwd_bwd     one mini-batch slice (128 samples) per cluster of 1, 2 or 4 blocks: forward (ReLU,
//                     sigmoid), mean binary cross-entropy gradient; activations and deltas staged in
//                     shared memory, partial gradients per slice (fixed summation order)
//   k_mlp_adam        sums the partials in block order and applies one Adam step
//   k_mlp_infer       inference, FP32 or BF16 (BF16 weights, inputs and hidden activations,
//                     FP32 accumulation)
//   k_mlp_accept      probability > threshold (or the ratio test when no network is given)
//                     -> (target, distance) rows for the one-to-one filter
//
// Parameter vector (float32): W1[64][8], b1[64], W2[64][64], b2[64], w3[64], b3, then the input
// normalisation mu[8], sigma[8] (not trained).
#include <cooperative_groups.h>
#include <cub/cub.cuh>
#include <cuda_bf16.h>

#include <cmath>
#include <vector>

#include "fsb_internal.cuh"

namespace fsb {
namespace {

constexpr int NF = 8, H = 64;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + H * NF, OFF_W2 = OFF_B1 + H, OFF_B2 = OFF_W2 + H * H,
              OFF_W3 = OFF_B2 + H, OFF_B3 = OFF_W3 + H, N_TRAIN = OFF_B3 + 1, OFF_MU = N_TRAIN,
              OFF_SIG = OFF_MU + NF, N_PARAM = OFF_SIG + NF;
constexpr int MB = 128;          // samples per slice (one partial gradient) of k_mlp_fwd_bwd
constexpr int HP = H + 4;        // row of the shared activation tiles: 16-byte rows, banks shifted by 4
constexpr int MT = 256;          // threads per block

inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// ------------------------------------------------------------------------ features
__global__ void k_mlp_features(int n, const int32_t* __restrict__ t1, const float* __restrict__ b12,
                               const double* __restrict__ pred, const float* __restrict__ xy_b,
                               const float* __restrict__ size_a, const float* __restrict__ angle_a,
                               const float* __restrict__ resp_a, const int32_t* __restrict__ oct_a,
                               const float* __restrict__ size_b, const float* __restrict__ angle_b,
                               const float* __restrict__ resp_b, float radius, float* __restrict__ feat) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float f[NF] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const int t = t1[i];
    if (t >= 0) {
        const float b1 = fmaxf(b12[2 * i], 0.f), b2 = b12[2 * i + 1];
        f[0] = isinf(b2) ? 0.f : sqrtf(b1) / fmaxf(sqrtf(fmaxf(b2, 0.f)), 1e-6f);
        f[1] = sqrtf(b1) * (1.f / 512.f);
        f[2] = log2f(fmaxf(size_b[t], 1e-6f) / fmaxf(size_a[i], 1e-6f));
        float da = angle_b[t] - angle_a[i];
        da = da - 360.f * floorf((da + 180.f) / 360.f);
        f[3] = da * (1.f / 180.f);
        const double dx = pred[2 * i] - (double)xy_b[2 * t], dy = pred[2 * i + 1] - (double)xy_b[2 * t + 1];
        f[4] = (float)sqrt(dx * dx + dy * dy) / radius;
        f[5] = resp_a[i];
        f[6] = resp_b[t];
        f[7] = (float)oct_a[i];
    }
#pragma unroll
    for (int k = 0; k < NF; ++k) feat[(size_t)i * NF + k] = f[k];
}

// ------------------------------------------------------------------------ training
__device__ __forceinline__ float sigmoidf_(float z) { return 1.f / (1.f + __expf(-z)); }

// acc[q][i] += sum over c = 0..63, in order, of W[c][i0 + i] * act[s_q][c] for NS samples s_q = s0 + 16 q
// and four outputs (W rows of pitch WP, act rows of pitch HP; the chain of fused multiply-adds of
// each output is one after another, so the blocking changes no rounding). Per four c: four 16-byte
// loads of W, NS of the activations, 8 NS packed multiply-adds.
template <int NS, int WP>
__device__ __forceinline__ void mlp_tile(const float* __restrict__ W, const float* __restrict__ act, int s0, int i0,
                                         float2 (&acc)[NS][2]) {
#pragma unroll 2
    for (int c = 0; c < H; c += 4) {
        float4 w[4], h[NS];
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = *reinterpret_cast<const float4*>(W + (c + k) * WP + i0);
#pragma unroll
        for (int q = 0; q < NS; ++q) h[q] = *reinterpret_cast<const float4*>(act + (s0 + 16 * q) * HP + c);
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            const float hv[4] = {h[q].x, h[q].y, h[q].z, h[q].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 hh = make_float2(hv[k], hv[k]);
                acc[q][0] = __ffma2_rn(make_float2(w[k].x, w[k].y), hh, acc[q][0]);
                acc[q][1] = __ffma2_rn(make_float2(w[k].z, w[k].w), hh, acc[q][1]);
            }
        }
    }
}

// h1 rows of `n` samples from the normalised features: a = b1[i] + sum_k W1[i][k] x[k] in order, ReLU,
// rounded to BF16 with BF16
template <bool BF16>
__device__ __forceinline__ float mlp_act(float a) {
    a = fmaxf(a, 0.f);
    return BF16 ? __bfloat162float(__float2bfloat16_rn(a)) : a;
}
// (W1T: [feature][output]); put(sample, first output, four values) stores
template <bool BF16, class Put>
__device__ __forceinline__ void mlp_h1(const float* __restrict__ W1T, const float* __restrict__ B1,
                                       const float* __restrict__ X, int n, Put put) {
    const int i0 = 4 * (threadIdx.x & 15);
    const float4 b = *reinterpret_cast<const float4*>(B1 + i0);
    float4 w[NF];
#pragma unroll
    for (int k = 0; k < NF; ++k) w[k] = *reinterpret_cast<const float4*>(W1T + k * H + i0);
    for (int s = threadIdx.x >> 4; s < n; s += MT / 16) {
        const float4 xa = *reinterpret_cast<const float4*>(X + s * NF), xb = *reinterpret_cast<const float4*>(X + s * NF + 4);
        const float x[NF] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
        float4 a = b;
#pragma unroll
        for (int k = 0; k < NF; ++k) {
            a.x = fmaf(w[k].x, x[k], a.x);
            a.y = fmaf(w[k].y, x[k], a.y);
            a.z = fmaf(w[k].z, x[k], a.z);
            a.w = fmaf(w[k].w, x[k], a.w);
        }
        put(s, i0, make_float4(mlp_act<BF16>(a.x), mlp_act<BF16>(a.y), mlp_act<BF16>(a.z), mlp_act<BF16>(a.w)));
    }
}
// the weights in shared memory, W1 and W2 transposed (W2T rows of pitch HP); W2 too when wanted
template <bool BF16, bool KEEP_W2>
__device__ __forceinline__ void mlp_weights(const float* __restrict__ prm, float* __restrict__ W1T, float* __restrict__ B1,
                                            float* __restrict__ W2, float* __restrict__ W2T, float* __restrict__ B2,
                                            float* __restrict__ W3) {
    auto wgt = [](float w) { return BF16 ? __bfloat162float(__float2bfloat16_rn(w)) : w; };
    const int tid = threadIdx.x;
    float t1[H * NF / MT], t2[H * H / MT], b[3] = {0.f, 0.f, 0.f};   // every load in flight at once
#pragma unroll
    for (int k = 0; k < H * NF / MT; ++k) t1[k] = prm[OFF_W1 + tid + k * MT];
#pragma unroll
    for (int k = 0; k < H * H / MT; ++k) t2[k] = prm[OFF_W2 + tid + k * MT];
    if (tid < H) {
        b[0] = prm[OFF_B1 + tid];
        b[1] = prm[OFF_B2 + tid];
        b[2] = prm[OFF_W3 + tid];
    }
#pragma unroll
    for (int k = 0; k < H * NF / MT; ++k) {
        const int i = tid + k * MT;
        W1T[(i & (NF - 1)) * H + i / NF] = wgt(t1[k]);
    }
#pragma unroll
    for (int k = 0; k < H * H / MT; ++k) {
        const int i = tid + k * MT;
        if (KEEP_W2) W2[i] = t2[k];
        W2T[(i & (H - 1)) * HP + (i >> 6)] = wgt(t2[k]);
    }
    if (tid < H) {
        B1[tid] = b[0];
        B2[tid] = b[1];
        W3[tid] = wgt(b[2]);
    }
}
// h2 = act(b2 + W2 h1) of 16 NS samples (W2T: [input][output], pitch HP)
template <int NS, bool BF16, class Put>
__device__ __forceinline__ void mlp_h2(const float* __restrict__ W2T, const float* __restrict__ B2,
                                       const float* __restrict__ H1, Put put) {
    const int s0 = threadIdx.x >> 4, i0 = 4 * (threadIdx.x & 15);
    float2 acc[NS][2];
    const float4 b = *reinterpret_cast<const float4*>(B2 + i0);
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        acc[q][0] = make_float2(b.x, b.y);
        acc[q][1] = make_float2(b.z, b.w);
    }
    mlp_tile<NS, HP>(W2T, H1, s0, i0, acc);
#pragma unroll
    for (int q = 0; q < NS; ++q)
        put(s0 + 16 * q, i0, make_float4(mlp_act<BF16>(acc[q][0].x), mlp_act<BF16>(acc[q][0].y),
                                         mlp_act<BF16>(acc[q][1].x), mlp_act<BF16>(acc[q][1].y)));
}
// z = b3 + sum_i w3[i] h2[i], in order
__device__ __forceinline__ float mlp_z(const float* __restrict__ W3, float b3, const float* __restrict__ h2) {
    float z = b3;
#pragma unroll
    for (int i = 0; i < H; i += 4) {
        const float4 w = *reinterpret_cast<const float4*>(W3 + i), h = *reinterpret_cast<const float4*>(h2 + i);
        z = fmaf(w.x, h.x, z);
        z = fmaf(w.y, h.y, z);
        z = fmaf(w.z, h.z, z);
        z = fmaf(w.w, h.w, z);
    }
    return z;
}

// Shared memory of a training block (floats): the weights, then every activation and delta of the
// slice's 128 samples. A block of a cluster computes its own 128 / CS samples and stores what another
// block's gradients need into that block's shared memory too.
struct MlpSmem {
    static constexpr int W1 = 0, B1 = W1 + H * NF, W2 = B1 + H, W2T = W2 + H * H, B2 = W2T + H * HP, W3 = B2 + H,
                         X = W3 + H, H1 = X + MB * NF, H2 = H1 + MB * HP, D2 = H2 + MB * HP, D1 = D2 + MB * HP,
                         DZ = D1 + MB * HP, LOSS = DZ + MB, ONE = LOSS + MB, END = ONE + 4;
};

// Partial gradient of mean BCE over one slice of 128 of `count` samples (sample = idx[base + s], the
// identity when idx is null) per cluster of CS blocks; part has N_TRAIN floats per slice. loss_sum
// (nullable) accumulates the summed loss. Block r of a cluster runs samples 128 r / CS .. of the
// forward and backward passes, and once the blocks have exchanged activations and deltas, sums the
// gradients of rows 64 r / CS .. of W1 and W2 (and their biases and w3) over the slice's samples in
// order: every gradient is one chain over samples 0 .. 127 whatever CS is.
// Bound by latency: a step of 8192 samples is 64 slices, 3.6 MFLOP each, on 148 SMs. One thread per
// sample with two shared loads per multiply-add on 64 SMs took 82 us a step with its Adam update;
// blocked tiles on clusters of two take 16 us (the launch, the weights and the Adam update 6 of them).
template <int CS>
__global__ void __launch_bounds__(MT) k_mlp_fwd_bwd(const float* __restrict__ prm, const float* __restrict__ feat,
                                                    const float* __restrict__ label,
                                                    const int32_t* __restrict__ idx, int base, int count,
                                                    float inv_batch, float* __restrict__ part,
                                                    double* __restrict__ loss_sum) {
    using S = MlpSmem;
    constexpr int SPC = MB / CS, NS = SPC / 16;   // samples of this block; per thread of a 16 x 16 tile grid
    constexpr int NI = H / CS;                    // gradient rows of this block
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x;
    const int rank = CS > 1 ? (int)(blockIdx.x % CS) : 0, slice = blockIdx.x / CS;
    const int l0 = rank * SPC;                    // first sample of this block within the slice
    // the samples do not depend on the step before: they load while it finishes
    constexpr int XN = (SPC * NF + MT - 1) / MT;
    float xr[XN], yr = 0.f;
    cudaTriggerProgrammaticLaunchCompletion();
#pragma unroll
    for (int k = 0; k < XN; ++k) {
        const int e = tid + k * MT, gi = slice * MB + l0 + e / NF;
        xr[k] = 0.f;
        if (e < SPC * NF && gi < count) xr[k] = feat[(size_t)(idx ? idx[base + gi] : base + gi) * NF + (e & (NF - 1))];
    }
    if (tid < SPC) {
        const int gi = slice * MB + l0 + tid;
        if (gi < count) yr = label[idx ? idx[base + gi] : base + gi];
    }
    cudaGridDependencySynchronize();   // the parameters of the step before (no-op without that launch attribute)
    mlp_weights<false, true>(prm, sm + S::W1, sm + S::B1, sm + S::W2, sm + S::W2T, sm + S::B2, sm + S::W3);
    const float mu = prm[OFF_MU + (tid & (NF - 1))], sig = prm[OFF_SIG + (tid & (NF - 1))], b3 = prm[OFF_B3];
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    float* peer[CS];   // the shared memory of the cluster's blocks, this one's included
#pragma unroll
    for (int r = 0; r < CS; ++r) peer[r] = CS > 1 ? cl.map_shared_rank(sm, r) : sm;
    if constexpr (CS > 1) cl.sync();   // every block of the cluster runs: its shared memory may be written
    if (tid == 0) sm[S::ONE] = 1.f;
#pragma unroll
    for (int k = 0; k < XN; ++k) {   // feature e % 8 = tid % 8
        const int e = tid + k * MT, gi = slice * MB + l0 + e / NF;
        if (e < SPC * NF) {
            const float x = gi < count ? (xr[k] - mu) / sig : 0.f;
#pragma unroll
            for (int r = 0; r < CS; ++r) peer[r][S::X + l0 * NF + e] = x;
        }
    }
    __syncthreads();
    // h1 of every sample goes to every block; of h2, d2 and d1 each column to the block that sums its
    // gradients
    auto all = [&](int at, float4 v) {
#pragma unroll
        for (int r = 0; r < CS; ++r) *reinterpret_cast<float4*>(peer[r] + at) = v;
    };
    auto own = [&](int at, int col, float4 v) {
        *reinterpret_cast<float4*>(sm + at) = v;
        if (CS > 1 && col / NI != rank) *reinterpret_cast<float4*>(cl.map_shared_rank(sm, col / NI) + at) = v;
    };
    mlp_h1<false>(sm + S::W1, sm + S::B1, sm + S::X + l0 * NF, SPC,
                  [&](int s, int i, float4 v) { all(S::H1 + (l0 + s) * HP + i, v); });
    __syncthreads();
    mlp_h2<NS, false>(sm + S::W2T, sm + S::B2, sm + S::H1 + l0 * HP,
                      [&](int s, int i, float4 v) { own(S::H2 + (l0 + s) * HP + i, i, v); });
    __syncthreads();
    if (tid < SPC) {
        const int s = l0 + tid, gi = slice * MB + s;
        const bool live = gi < count;
        const float z = mlp_z(sm + S::W3, b3, sm + S::H2 + s * HP);
        const float y = yr;
        const float p = sigmoidf_(z);
        // BCE with logits: max(z, 0) - z y + log(1 + exp(-|z|))
        peer[0][S::LOSS + s] = live ? fmaxf(z, 0.f) - z * y + log1pf(__expf(-fabsf(z))) : 0.f;
        const float dz = live ? (p - y) * inv_batch : 0.f;
#pragma unroll
        for (int r = 0; r < CS; ++r) peer[r][S::DZ + s] = dz;
    }
    __syncthreads();
    for (int e = tid; e < SPC * (H / 4); e += MT) {
        const int s = l0 + (e >> 4), i0 = 4 * (e & 15);
        const float dz = sm[S::DZ + s];
        const float4 h = *reinterpret_cast<const float4*>(sm + S::H2 + s * HP + i0);
        const float4 w = *reinterpret_cast<const float4*>(sm + S::W3 + i0);
        own(S::D2 + s * HP + i0, i0,
            make_float4(h.x > 0.f ? dz * w.x : 0.f, h.y > 0.f ? dz * w.y : 0.f, h.z > 0.f ? dz * w.z : 0.f,
                        h.w > 0.f ? dz * w.w : 0.f));
    }
    __syncthreads();
    {   // d1[s][j] = sum_i W2[i][j] d2[s][i] where h1[s][j] > 0
        const int s0 = l0 + (tid >> 4), j0 = 4 * (tid & 15);
        float2 acc[NS][2];
#pragma unroll
        for (int q = 0; q < NS; ++q) acc[q][0] = acc[q][1] = make_float2(0.f, 0.f);
        mlp_tile<NS, H>(sm + S::W2, sm + S::D2, s0, j0, acc);
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            const float4 h = *reinterpret_cast<const float4*>(sm + S::H1 + (s0 + 16 * q) * HP + j0);
            own(S::D1 + (s0 + 16 * q) * HP + j0, j0,
                make_float4(h.x > 0.f ? acc[q][0].x : 0.f, h.y > 0.f ? acc[q][0].y : 0.f, h.z > 0.f ? acc[q][1].x : 0.f,
                            h.w > 0.f ? acc[q][1].y : 0.f));
        }
    }
    if constexpr (CS > 1) cl.sync();   // every block's stores have landed; no remote access after this
    else __syncthreads();
    float* out = part + (size_t)slice * N_TRAIN;
    const int ib = rank * NI;
    if (tid < 128) {
        // W2[i][j] = sum_s d2[s][i] h1[s][j], s in order: TI rows x four columns per thread
        constexpr int TI = NI / 8;
        const int i0 = ib + (tid >> 4) * TI, j0 = 4 * (tid & 15);
        float2 g[TI][2];
#pragma unroll
        for (int i = 0; i < TI; ++i) g[i][0] = g[i][1] = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int q = 0; q < MB; ++q) {
            const float4 h = *reinterpret_cast<const float4*>(sm + S::H1 + q * HP + j0);
            float d[TI];
            const float* dp = sm + S::D2 + q * HP + i0;
            if constexpr (TI % 4 == 0) {
#pragma unroll
                for (int i = 0; i < TI; i += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(dp + i);
                    d[i] = v.x;
                    d[i + 1] = v.y;
                    d[i + 2] = v.z;
                    d[i + 3] = v.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < TI; ++i) d[i] = dp[i];
            }
#pragma unroll
            for (int i = 0; i < TI; ++i) {
                g[i][0] = __ffma2_rn(make_float2(d[i], d[i]), make_float2(h.x, h.y), g[i][0]);
                g[i][1] = __ffma2_rn(make_float2(d[i], d[i]), make_float2(h.z, h.w), g[i][1]);
            }
        }
#pragma unroll
        for (int i = 0; i < TI; ++i) {
            float* o = out + OFF_W2 + (i0 + i) * H + j0;   // N_TRAIN is odd: no wide stores
            o[0] = g[i][0].x;
            o[1] = g[i][0].y;
            o[2] = g[i][1].x;
            o[3] = g[i][1].y;
        }
    } else {
        // The others, all chains of a thread in one branch-free sweep (so that the loads of several
        // samples are in flight): W1[i][k] = sum d1 x for KN features; and EX of b1 = sum 1 d1,
        // b2 = sum 1 d2, w3 = sum dz h2, b3 = sum dz 1 (a multiply-add by one rounds like an addition).
        constexpr int G = 128 / NI;                     // groups of NI threads
        constexpr int KN = G >= NF ? 1 : NF / G, EX = G >= 4 ? 1 : 4 / G;
        const int u = tid - 128, i = ib + u % NI, grp = u / NI, k0 = grp * KN;
        const float *pa[EX], *pb[EX];
        int sa[EX], sb[EX], what[EX];
#pragma unroll
        for (int x = 0; x < EX; ++x) {
            what[x] = grp * EX + x;
            pa[x] = pb[x] = sm + S::ONE;
            sa[x] = sb[x] = 0;
            if (what[x] == 0) pb[x] = sm + S::D1 + i;
            if (what[x] == 1) pb[x] = sm + S::D2 + i;
            if (what[x] == 2) pb[x] = sm + S::H2 + i;
            if (what[x] <= 2) sb[x] = HP;
            if (what[x] == 2 || what[x] == 3) {
                pa[x] = sm + S::DZ;
                sa[x] = 1;
            }
        }
        const float* px = sm + S::X + min(k0, NF - KN);
        const float* pd = sm + S::D1 + i;
        float g[KN], ge[EX];
#pragma unroll
        for (int k = 0; k < KN; ++k) g[k] = 0.f;
#pragma unroll
        for (int x = 0; x < EX; ++x) ge[x] = 0.f;
#pragma unroll 8
        for (int q = 0; q < MB; ++q) {
            const float d1 = pd[q * HP];
#pragma unroll
            for (int k = 0; k < KN; ++k) g[k] = fmaf(d1, px[q * NF + k], g[k]);
#pragma unroll
            for (int x = 0; x < EX; ++x) ge[x] = fmaf(pa[x][q * sa[x]], pb[x][q * sb[x]], ge[x]);
        }
        if (k0 < NF) {
#pragma unroll
            for (int k = 0; k < KN; ++k) out[OFF_W1 + i * NF + k0 + k] = g[k];
        }
#pragma unroll
        for (int x = 0; x < EX; ++x) {
            if (what[x] == 0) out[OFF_B1 + i] = ge[x];
            if (what[x] == 1) out[OFF_B2 + i] = ge[x];
            if (what[x] == 2) out[OFF_W3 + i] = ge[x];
            if (what[x] == 3 && i == 0) out[OFF_B3] = ge[x];
        }
    }
    if (loss_sum && rank == 0 && tid < 32) {
        // sums of 32 samples by lane pairs, the four sums in order
        float l = 0.f;
        for (int w = 0; w < MB / 32; ++w) {
            float v = sm[S::LOSS + 32 * w + tid];
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            l += v;
        }
        if (tid == 0) atomicAdd(loss_sum, (double)l);
    }
}

// Sum of the partial gradients (slice order) and Adam step number t (from 1).
constexpr int AT = 64;   // threads per block: 75 blocks for the 4 737 parameters
__global__ void __launch_bounds__(AT) k_mlp_adam(float* __restrict__ prm, float* __restrict__ m, float* __restrict__ v,
                                                 const float* __restrict__ part, int nparts,
                                                 int t, float lr, float* __restrict__ grad_out) {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= N_TRAIN) return;
    float g = 0.f;
    int b = 0;
    for (; b + 32 <= nparts; b += 32) {   // 32 loads in flight, added in order
        float p[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) p[k] = part[(size_t)(b + k) * N_TRAIN + e];
#pragma unroll
        for (int k = 0; k < 32; ++k) g += p[k];
    }
    for (; b < nparts; ++b) g += part[(size_t)b * N_TRAIN + e];
    if (grad_out) grad_out[e] = g;
    if (!m) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mm = b1 * m[e] + (1.f - b1) * g;
    const float vv = b2 * v[e] + (1.f - b2) * g * g;
    m[e] = mm;
    v[e] = vv;
    const float mh = mm / (1.f - powf(b1, (float)t)), vh = vv / (1.f - powf(b2, (float)t));
    prm[e] -= lr * mh / (sqrtf(vh) + eps);
}

__global__ void k_mlp_perm_keys(int n, int epoch, uint32_t seed, uint32_t* __restrict__ key,
                                int32_t* __restrict__ val) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // splitmix-style 32-bit hash of (seed, epoch, i)
    uint32_t h = seed ^ (0x9E3779B9u * (uint32_t)(epoch + 1)) ^ (0x85EBCA6Bu * (uint32_t)i);
    h ^= h >> 16;
    h *= 0x7FEB352Du;
    h ^= h >> 15;
    h *= 0x846CA68Bu;
    h ^= h >> 16;
    key[i] = h;
    val[i] = i;
}

// ------------------------------------------------------------------------ inference
__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// Inference of 128 samples per block and step (blocks walk the samples): the training pass's tiles, so
// every pre-activation is the same chain of multiply-adds. Bound by the multiply-adds (4 672 a sample);
// one thread per sample with a shared load per multiply-add took 223 us for 390 000 samples, the
// tiles take 100 us.
struct InferSmem {
    static constexpr int W1 = 0, B1 = W1 + H * NF, W2T = B1 + H, B2 = W2T + H * HP, W3 = B2 + H, X = W3 + H,
                         H1 = X + MB * NF, H2 = H1 + MB * HP, END = H2 + MB * HP;
};
template <bool BF16>
__global__ void __launch_bounds__(MT, 2) k_mlp_infer(const float* __restrict__ prm, int n, const float* __restrict__ feat,
                                                     float* __restrict__ prob) {
    using S = InferSmem;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x;
    mlp_weights<BF16, false>(prm, sm + S::W1, sm + S::B1, nullptr, sm + S::W2T, sm + S::B2, sm + S::W3);
    const float b3 = prm[OFF_B3];
    const float mu = prm[OFF_MU + (tid & 7)], sig = prm[OFF_SIG + (tid & 7)];
    const int tiles = (n + MB - 1) / MB;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int base = t * MB;
        __syncthreads();   // the previous tile's rows are done (first pass: the weights)
#pragma unroll
        for (int e = tid; e < MB * NF; e += MT) {   // k = e % 8 = tid % 8
            float x = 0.f;
            if (base + (e >> 3) < n) x = (feat[(size_t)base * NF + e] - mu) / sig;
            sm[S::X + e] = BF16 ? bf16r(x) : x;
        }
        __syncthreads();
        mlp_h1<BF16>(sm + S::W1, sm + S::B1, sm + S::X, MB, [&](int s, int i, float4 v) {
            *reinterpret_cast<float4*>(sm + S::H1 + s * HP + i) = v;
        });
        __syncthreads();
        mlp_h2<MB / 16, BF16>(sm + S::W2T, sm + S::B2, sm + S::H1, [&](int s, int i, float4 v) {
            *reinterpret_cast<float4*>(sm + S::H2 + s * HP + i) = v;
        });
        __syncthreads();
        if (tid < MB && base + tid < n) prob[base + tid] = sigmoidf_(mlp_z(sm + S::W3, b3, sm + S::H2 + tid * HP));
    }
}

__global__ void k_mlp_accept(int n, const int32_t* __restrict__ t1, const float* __restrict__ b12,
                             const float* __restrict__ prob, float thr, float ratio, int32_t* __restrict__ t_row,
                             uint32_t* __restrict__ d_row) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int t = t1[i];
    bool ok = false;
    if (t >= 0) {
        if (prob) {
            ok = prob[i] > thr;
        } else {   // plain ratio test (app/planesite/matching.py:142-146; a single candidate passes)
            ok = __fsqrt_rn(fmaxf(b12[2 * i], 0.f)) < __fmul_rn(ratio, __fsqrt_rn(b12[2 * i + 1]));
        }
    }
    t_row[i] = ok ? t : -1;
    d_row[i] = ok ? (uint32_t)b12[2 * i] : 0u;
}

template <int CS>
int32_t launch_fwd_bwd_t(int slices, const float* prm, const float* feat, const float* label, const int32_t* idx, int base,
                         int count, float inv_batch, float* part, double* loss, bool overlap, cudaStream_t s) {
    static std::atomic<int> done[64];
    constexpr int bytes = MlpSmem::END * 4;
    FSB_TRY(smem_attr((const void*)k_mlp_fwd_bwd<CS>, bytes, done));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)slices * CS);
    cfg.blockDim = dim3(MT);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    int na = 0;
    if (CS > 1) {
        at[na].id = cudaLaunchAttributeClusterDimension;
        at[na].val.clusterDim.x = CS;
        at[na].val.clusterDim.y = 1;
        at[na++].val.clusterDim.z = 1;
    }
    if (overlap) {
        at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[na++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = na;
    FSB_CUDA(cudaLaunchKernelEx(&cfg, k_mlp_fwd_bwd<CS>, prm, feat, label, idx, base, count, inv_batch, part, loss));
    note_launch();
    return FSB_OK;
}
// blocks per slice: as many as keep every slice resident at once (one block per SM), at most four
// (clusters of eight such blocks find few places: 55 us a step of 2048 against 13 with four).
// overlap: the launch may start while the kernel before it (an Adam step, which nothing but the
// parameters and the partials of this kernel depend on) is running
int32_t launch_fwd_bwd(int slices, const float* prm, const float* feat, const float* label, const int32_t* idx, int base,
                       int count, float inv_batch, float* part, double* loss, bool overlap, cudaStream_t s) {
    auto* f = slices * 4 <= 128 ? launch_fwd_bwd_t<4> : slices * 2 <= 140 ? launch_fwd_bwd_t<2> : launch_fwd_bwd_t<1>;
    return f(slices, prm, feat, label, idx, base, count, inv_batch, part, loss, overlap, s);
}
int32_t launch_adam(float* prm, float* m, float* v, const float* part, int nparts, int t, float lr, float* grad,
                    cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nblk(N_TRAIN, AT));
    cfg.blockDim = dim3(AT);
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    FSB_CUDA(cudaLaunchKernelEx(&cfg, k_mlp_adam, prm, m, v, part, nparts, t, lr, grad));
    note_launch();
    return FSB_OK;
}
template <bool BF16>
int32_t launch_infer(const float* prm, int n, const float* feat, float* prob, cudaStream_t s) {
    static std::atomic<int> done[64];
    constexpr int bytes = InferSmem::END * 4;
    FSB_TRY(smem_attr((const void*)k_mlp_infer<BF16>, bytes, done));
    k_mlp_infer<BF16><<<std::min(nblk(n, MB), 2u * 148u), MT, bytes, s>>>(prm, n, feat, prob);
    note_launch();
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}

}  // namespace

int mlp_param_count() { return N_PARAM; }
int mlp_trainable_count() { return N_TRAIN; }

int32_t run_mlp_features(int n, const int32_t* t1, const float* b12, const double* pred, const float* xy_b,
                         const float* size_a, const float* angle_a, const float* resp_a, const int32_t* oct_a,
                         const float* size_b, const float* angle_b, const float* resp_b, float radius, float* feat,
                         cudaStream_t s) {
    if (n <= 0) return FSB_OK;
    k_mlp_features<<<nblk(n, 256), 256, 0, s>>>(n, t1, b12, pred, xy_b, size_a, angle_a, resp_a, oct_a, size_b,
                                                angle_b, resp_b, radius, feat);
    note_launch();
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}

int32_t run_mlp_infer(const float* prm, int n, const float* feat, bool bf16, float* prob, cudaStream_t s) {
    if (n <= 0) return FSB_OK;
    return bf16 ? launch_infer<true>(prm, n, feat, prob, s) : launch_infer<false>(prm, n, feat, prob, s);
}

int32_t run_mlp_accept(int n, const int32_t* t1, const float* b12, const float* prob, float thr, float ratio,
                       int32_t* t_row, uint32_t* d_row, cudaStream_t s) {
    if (n <= 0) return FSB_OK;
    k_mlp_accept<<<nblk(n, 256), 256, 0, s>>>(n, t1, b12, prob, thr, ratio, t_row, d_row);
    note_launch();
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}

// Mean-BCE gradient over samples idx[0..n) (identity when idx is null) into grad (N_TRAIN floats).
int32_t run_mlp_grad(fsb_ctx* ctx, const float* prm, int n, const float* feat, const float* label, float* grad,
                     double* loss, cudaStream_t s) {
    const int nb = (int)nblk(n, MB);
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    FSB_TRY(ctx->s_misc.ensure(al((size_t)nb * N_TRAIN * 4) + al(64)));
    uint8_t* base = ctx->s_misc.as<uint8_t>();
    float* part = reinterpret_cast<float*>(base);
    double* dl = reinterpret_cast<double*>(base + al((size_t)nb * N_TRAIN * 4));
    FSB_CUDA(cudaMemsetAsync(dl, 0, 8, s));
    FSB_TRY(launch_fwd_bwd(nb, prm, feat, label, nullptr, 0, n, 1.f / (float)n, part, dl, false, s));
    FSB_TRY(launch_adam(nullptr, nullptr, nullptr, part, nb, 0, 0.f, grad, s));
    FSB_CUDA(cudaGetLastError());
    double h = 0.0;
    FSB_CUDA(cudaMemcpyAsync(&h, dl, 8, cudaMemcpyDeviceToHost, s));
    FSB_CUDA(cudaStreamSynchronize(s));
    if (loss) *loss = h / (double)n;
    return FSB_OK;
}

// Mini-batch Adam over n samples for `epochs` epochs. prm (N_PARAM), m, v (N_TRAIN) in device memory.
// Each epoch: shuffle (hash keys + radix sort), then floor(n / batch) steps (one step of n when
// n < batch). Two launches a step, queued without a host wait until the end; each may start while the
// one before it drains (the samples of a step load during the Adam step before it). losses (host,
// nullable, `epochs` entries) receives the mean training loss of every epoch.
int32_t run_mlp_train(fsb_ctx* ctx, float* prm, float* m, float* v, int n, const float* feat, const float* label,
                      int epochs, int batch, float lr, uint32_t seed, double* losses, cudaStream_t s) {
    batch = std::max(MB, (batch / MB) * MB);
    const int bsz = n < batch ? n : batch;
    const int steps = n < batch ? 1 : n / batch;
    const int nb = (int)nblk(bsz, MB);
    size_t tb = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tb, (uint32_t*)nullptr, (uint32_t*)nullptr, (int32_t*)nullptr,
                                    (int32_t*)nullptr, n, 0, 32, s);
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    if (epochs < 0) epochs = 0;
    const size_t need = al((size_t)nb * N_TRAIN * 4) + 4 * al((size_t)n * 4) + al(tb) + al((size_t)epochs * 8 + 8);
    FSB_TRY(ctx->s_misc.ensure(need));
    uint8_t* cur = ctx->s_misc.as<uint8_t>();
    auto take = [&](size_t bytes) {
        uint8_t* p = cur;
        cur += (bytes + 255) & ~size_t(255);
        return p;
    };
    float* part = reinterpret_cast<float*>(take((size_t)nb * N_TRAIN * 4));
    uint32_t* keys = reinterpret_cast<uint32_t*>(take((size_t)n * 4));
    uint32_t* keys2 = reinterpret_cast<uint32_t*>(take((size_t)n * 4));
    int32_t* vals = reinterpret_cast<int32_t*>(take((size_t)n * 4));
    int32_t* perm = reinterpret_cast<int32_t*>(take((size_t)n * 4));
    void* tmp = take(tb);
    double* dl = reinterpret_cast<double*>(take((size_t)epochs * 8 + 8));   // loss sums of the epochs
    FSB_CUDA(cudaMemsetAsync(dl, 0, (size_t)epochs * 8 + 8, s));
    FSB_CUDA(cudaMemsetAsync(m, 0, (size_t)N_TRAIN * 4, s));
    FSB_CUDA(cudaMemsetAsync(v, 0, (size_t)N_TRAIN * 4, s));
    for (int e = 0; e < epochs; ++e) {
        k_mlp_perm_keys<<<nblk(n, 256), 256, 0, s>>>(n, e, seed, keys, vals);
        size_t tbe = tb;
        FSB_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tbe, keys, keys2, vals, perm, n, 0, 32, s));
        note_launch(2);
        for (int st = 0; st < steps; ++st) {
            FSB_TRY(launch_fwd_bwd(nb, prm, feat, label, perm, st * bsz, bsz, 1.f / (float)bsz, part, dl + e, st > 0, s));
            FSB_TRY(launch_adam(prm, m, v, part, nb, e * steps + st + 1, lr, nullptr, s));
        }
    }
    FSB_CUDA(cudaGetLastError());
    std::vector<double> h(epochs > 0 ? epochs : 1, 0.0);
    if (losses && epochs > 0)
        FSB_CUDA(cudaMemcpyAsync(h.data(), dl, (size_t)epochs * 8, cudaMemcpyDeviceToHost, s));
    FSB_CUDA(cudaStreamSynchronize(s));
    for (int e = 0; losses && e < epochs; ++e) losses[e] = h[e] / ((double)steps * bsz);
    return FSB_OK;
}

}  // namespace fsb
