// The learned warm start of the FEM step's PCG solve: a per-node MLP 36 -> 64 -> 64 -> 64 -> 12 (ReLU), BF16 weights
// with FP32 accumulation, its inference in the step, the recording of training samples from the Cholesky's solves,
// and its training (forward, backward, Adam) on the GPU. No counterpart in the reference.
//
// Features of a frame node i (column k = iperm[i]), with sl(x) = sign(x) log(1 + |x| / s0), s0 = 1 mm/s:
//   0-2   sl(h F_i / m_i)             the explicit step's velocity change (F: the node's force before the solve)
//   3-5   sl(dv_i of the last solve)
//   6-8   sl(v_i)
//   9-11  the mean of features 0-2 over the node's 1-ring (the frame nodes it shares a triangle with)
//   12-14 the mean of features 3-5 over the 1-ring
//   15-32 the edges to the first six 1-ring nodes (in frame-node order), (x_j - x_i) / their mean length; zeros after
//   33-35 log(D_aa / m_i): the translational diagonal of the node's 6 x 6 diagonal block of A over its mass
// Outputs: y 0-2 -> the guess dv = isl(y) (the inverse of sl); y 3-11 -> S = I + 0.25 tanh(y) entrywise (3 x 3, row
// major): the preconditioner's translational scale (bl_fem_pcg.cuh).
// Training targets (recorded from the Cholesky's solutions): sl(dv) for y 0-2; for the diagonal of S the ratio of the
// solution to the block-Jacobi estimate u = (D^-1 rhs)_a, clamped to [0.76, 1.24] (weight 0.1 where |u_a| > 1e-9 m/s),
// zero for its off-diagonal entries (weight 0.01).
//
// Parameters, one float vector: W1 (64 x 36, row = output), b1 (64), W2 (64 x 64), b2, W3 (64 x 64), b3, W4 (12 x 64), b4.
// The forward's four layers run on the tensor cores (mma.sync m16n8k16, BF16 inputs and weights, FP32 accumulation,
// FP32 bias and ReLU; each layer's input rounded to BF16); the backward (data and weight gradients) runs in FP32 on the
// BF16-rounded activations the forward used.
#pragma once

#include <cuda_bf16.h>

#include "bl_fem_kernels.cuh"

namespace blg {

constexpr int kIn = 36, kHid = 64, kOut = 12;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kHid * kIn, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid, kOffW3 = kOffB2 + kHid;
constexpr int kOffB3 = kOffW3 + kHid * kHid, kOffW4 = kOffB3 + kHid, kOffB4 = kOffW4 + kOut * kHid, kParams = kOffB4 + kOut;
constexpr float kS0 = 1e-3f;

struct MlpDev {
    const __nv_bfloat16* wb; // the parameters in BF16 (what the forward reads)
    float* w;                // FP32 master copy (what Adam updates)
    float* m;                // Adam moments
    float* v;
    // the step's side
    const int* adj_ptr;      // per frame node: its 1-ring (frame nodes sharing a triangle), ascending
    const int* adj;
    float* prev_dv;          // 3 / frame node: dv of the last solve
    float* feat;             // kIn / frame node: this substep's features
    // recorded samples (a ring of cap samples)
    float* sx;               // kIn / sample
    float* st;               // kOut / sample: targets
    float* sw;               // kOut / sample: weights
    int* scount;             // samples recorded so far
    int cap;
};

__device__ __forceinline__ float slog(float x) { return x < 0 ? -log1pf(-x / kS0) : log1pf(x / kS0); }
__device__ __forceinline__ float islog(float y) { return y < 0 ? -kS0 * expm1f(-y) : kS0 * expm1f(y); }

// ------------------------------------------------------------------------------------------ the network
// A block of 8 warps takes tiles of 32 samples; a layer is 32 samples x 64 outputs as mma.sync m16n8k16 tiles (BF16
// operands, FP32 accumulation), a warp one column of 8 outputs: A = the layer's input, 32 rows of BF16 in shared memory
// (row stride kPadIn: rows fall in distinct banks), B = the weights, kept in the warp's registers over all its tiles. The
// inputs are rounded to BF16 as they are staged (the activations the next layer reads are the BF16 values); the
// accumulators, bias and ReLU stay FP32.
constexpr int kTile = 32;        // samples a tile
constexpr int kMlpThreads = 256;
constexpr int kPadIn = 64 + 8;   // a BF16 row
constexpr int kPadF = 64 + 4;    // an FP32 row

__device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t lds32(const __nv_bfloat16* p) { return *reinterpret_cast<const uint32_t*>(p); }

// a tile's activations: act - the current layer's input and the next one's, BF16; a - each layer's input as FP32 of the
// BF16 values (what the weight gradients multiply); y - the outputs
struct MlpTile {
    __nv_bfloat16 act[2][kTile * kPadIn];
    float a[4][kTile * kPadF];
    float y[kTile * 16];
};

// a warp's weights: its 8 outputs of each layer (k-steps of 16; zero past the layer's inputs and outputs) and biases
struct MlpFrag {
    uint32_t w[4][4][2];
    float b[4][2];
};
__device__ __forceinline__ void mlp_load(const __nv_bfloat16* __restrict__ wb, MlpFrag& W) {
    const int lane = threadIdx.x & 31, nt = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int offw[4] = {kOffW1, kOffW2, kOffW3, kOffW4}, offb[4] = {kOffB1, kOffB2, kOffB3, kOffB4};
#pragma unroll
    for (int l = 0; l < 4; l++) {
        const int nin = l == 0 ? kIn : kHid, nout = l == 3 ? kOut : kHid, o = 8 * nt + g;
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int i = 16 * k + 8 * h + 2 * t; // (even, as nin: a pair is inside or outside)
                W.w[l][k][h] = o < nout && i < nin ? *reinterpret_cast<const uint32_t*>(wb + offw[l] + (size_t)o * nin + i) : 0u;
            }
#pragma unroll
        for (int h = 0; h < 2; h++) W.b[l][h] = 8 * nt + 2 * t + h < nout ? __bfloat162float(wb[offb[l] + 8 * nt + 2 * t + h]) : 0.0f;
    }
}

// The forward of a tile: x(sample, feature) its features. Ends with y in place and the block synchronised.
template <class X>
__device__ __forceinline__ void mlp_forward(const MlpFrag& W, MlpTile& S, X x) {
    const int lane = threadIdx.x & 31, nt = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    for (int e = threadIdx.x; e < kTile * 48; e += kMlpThreads) { // (36 features, zeros to three k-steps)
        const int smp = e / 48, i = e % 48;
        const __nv_bfloat16 v = __float2bfloat16(i < kIn ? x(smp, i) : 0.0f);
        S.act[0][smp * kPadIn + i] = v;
        if (i < kIn) S.a[0][smp * kPadF + i] = __bfloat162float(v);
    }
    __syncthreads();
#pragma unroll
    for (int l = 0; l < 4; l++) {
        const __nv_bfloat16* in = S.act[l & 1];
        if (l < 3 || nt < 2) {
            float c[2][4];
#pragma unroll
            for (int mt = 0; mt < 2; mt++)
#pragma unroll
                for (int q = 0; q < 4; q++) c[mt][q] = 0.0f;
#pragma unroll
            for (int k = 0; k < (l == 0 ? 3 : 4); k++)
#pragma unroll
                for (int mt = 0; mt < 2; mt++) {
                    const __nv_bfloat16* lo = in + (16 * mt + g) * kPadIn + 16 * k + 2 * t;
                    const __nv_bfloat16* hi = lo + 8 * kPadIn;
                    const uint32_t a[4] = {lds32(lo), lds32(hi), lds32(lo + 8), lds32(hi + 8)};
                    mma_bf16(c[mt], a, W.w[l][k][0], W.w[l][k][1]);
                }
            // c0, c1: sample 16 mt + g, outputs 8 nt + 2 t, + 1; c2, c3: sample + 8
#pragma unroll
            for (int mt = 0; mt < 2; mt++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int smp = 16 * mt + g + (q >= 2 ? 8 : 0), o = 8 * nt + 2 * t + (q & 1);
                    const float v = c[mt][q] + W.b[l][q & 1];
                    if (l == 3) {
                        S.y[smp * 16 + o] = v;
                    } else {
                        const __nv_bfloat16 r = __float2bfloat16(fmaxf(v, 0.0f));
                        S.act[(l + 1) & 1][smp * kPadIn + o] = r;
                        S.a[l + 1][smp * kPadF + o] = __bfloat162float(r);
                    }
                }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------ the step's side
// The features of every frame node (after the assembly: diag holds A's diagonal blocks, nforce the nodes' forces)
__global__ void k_mlp_features(FemDev F, MlpDev M, const float4* __restrict__ nd, const float4* __restrict__ nforce) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= F.nf) return;
    float* x = M.feat + (size_t)kIn * i;
    auto explicit_dv = [&](int j, float* e) {
        const int bn = F.fnode[j];
        const float4 f = nforce[bn];
        const float m = nd[2 * bn + 1].w;
        const float s = m > 0 ? F.h / m : 0.0f;
        e[0] = slog(f.x * s), e[1] = slog(f.y * s), e[2] = slog(f.z * s);
    };
    float e[3];
    explicit_dv(i, e);
    const int bn = F.fnode[i];
    const float4 P = nd[2 * bn], Vv = nd[2 * bn + 1];
    for (int a = 0; a < 3; a++) x[a] = e[a], x[3 + a] = slog(M.prev_dv[3 * i + a]);
    x[6] = slog(Vv.x), x[7] = slog(Vv.y), x[8] = slog(Vv.z);
    float me[3] = {0, 0, 0}, mp[3] = {0, 0, 0};
    const int j0 = M.adj_ptr[i], j1 = M.adj_ptr[i + 1];
    float mean_len = 0;
    for (int q = j0; q < j1; q++) {
        const int j = M.adj[q];
        float ej[3];
        explicit_dv(j, ej);
        for (int a = 0; a < 3; a++) me[a] += ej[a], mp[a] += slog(M.prev_dv[3 * j + a]);
        const float4 Pj = nd[2 * F.fnode[j]];
        mean_len += sqrtf((Pj.x - P.x) * (Pj.x - P.x) + (Pj.y - P.y) * (Pj.y - P.y) + (Pj.z - P.z) * (Pj.z - P.z));
    }
    const int nn = j1 - j0;
    const float inv = nn > 0 ? 1.0f / (float)nn : 0.0f;
    for (int a = 0; a < 3; a++) x[9 + a] = me[a] * inv, x[12 + a] = mp[a] * inv;
    mean_len = nn > 0 ? mean_len * inv : 1.0f;
    const float il = mean_len > 0 ? 1.0f / mean_len : 0.0f;
    for (int q = 0; q < 6; q++) {
        if (q < nn) {
            const float4 Pj = nd[2 * F.fnode[M.adj[j0 + q]]];
            x[15 + 3 * q] = (Pj.x - P.x) * il, x[16 + 3 * q] = (Pj.y - P.y) * il, x[17 + 3 * q] = (Pj.z - P.z) * il;
        } else {
            x[15 + 3 * q] = x[16 + 3 * q] = x[17 + 3 * q] = 0.0f;
        }
    }
    const int k = F.iperm[i];
    const double* D = F.diag + 36 * (size_t)k;
    const float m = Vv.w;
    for (int a = 0; a < 3; a++) x[33 + a] = (m > 0 && !(P.w <= 0)) ? logf(fmaxf((float)(D[a * 7] / (double)m), 1e-6f)) : 0.0f;
}

// The network on every frame node's features: the PCG's guess and scale
__global__ void __launch_bounds__(kMlpThreads) k_mlp_infer(FemDev F, MlpDev M, float* __restrict__ guess, float* __restrict__ gscale) {
    __shared__ __align__(16) MlpTile S;
    MlpFrag W;
    mlp_load(M.wb, W);
    const int i0 = blockIdx.x * kTile;
    mlp_forward(W, S, [&](int smp, int f) { return i0 + smp < F.nf ? M.feat[(size_t)kIn * (i0 + smp) + f] : 0.0f; });
    for (int e = threadIdx.x; e < kTile * kOut; e += kMlpThreads) {
        const int i = i0 + e / kOut, q = e % kOut;
        if (i >= F.nf) continue;
        const float y = S.y[(e / kOut) * 16 + q];
        if (q < 3) guess[3 * i + q] = islog(y);
        else gscale[9 * i + q - 3] = (((q - 3) % 4) == 0 ? 1.0f : 0.0f) + 0.25f * tanhf(y);
    }
}

// Recording, before the solve: each frame node's features and the block-Jacobi estimate u = (D^-1 rhs)_a (kept in
// the targets' slots 3-5 until k_mlp_record_post)
__global__ void k_mlp_record_pre(FemDev F, MlpDev M) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= F.nf) return;
    const size_t slot = (size_t)((*M.scount + i) % M.cap);
    for (int f = 0; f < kIn; f++) M.sx[kIn * slot + f] = M.feat[(size_t)kIn * i + f];
    const int k = F.iperm[i];
    double L[36], di[6], u[6];
    for (int x = 0; x < 36; x++) L[x] = F.diag[36 * (size_t)k + x];
    for (int j = 0; j < 6; j++) u[j] = F.rhs[6 * (size_t)k + j];
    if (chol6_dev(L, di)) {
        for (int j = 0; j < 6; j++) {
            double t = u[j];
            for (int m = 0; m < j; m++) t -= L[j * 6 + m] * u[m];
            u[j] = t * di[j];
        }
        for (int j = 5; j >= 0; j--) {
            double t = u[j];
            for (int m = j + 1; m < 6; m++) t -= L[m * 6 + j] * u[m];
            u[j] = t * di[j];
        }
    } else {
        for (int j = 0; j < 6; j++) u[j] = 0.0;
    }
    for (int a = 0; a < 3; a++) M.st[kOut * slot + 3 + a] = (float)u[a];
}

// Recording, after the solve: the targets from the solution dv (in rhs) and u
__global__ void k_mlp_record_post(FemDev F, MlpDev M) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= F.nf) return;
    const size_t slot = (size_t)((*M.scount + i) % M.cap);
    const int k = F.iperm[i];
    const bool fixed = F.fixed[k] != 0;
    float* t = M.st + kOut * slot;
    float* w = M.sw + kOut * slot;
    float u[3];
    for (int a = 0; a < 3; a++) u[a] = t[3 + a];
    for (int a = 0; a < 3; a++) {
        const float dv = (float)F.rhs[6 * (size_t)k + a];
        t[a] = slog(dv), w[a] = fixed ? 0.0f : 1.0f;
    }
    for (int q = 0; q < 9; q++) {
        const int r = q / 3, c = q % 3;
        if (r == c) {
            const float dv = (float)F.rhs[6 * (size_t)k + r];
            const bool ok = !fixed && fabsf(u[r]) > 1e-9f;
            const float ratio = ok ? fminf(fmaxf(dv / u[r], 0.76f), 1.24f) : 1.0f;
            t[3 + q] = atanhf((ratio - 1.0f) / 0.25f);
            w[3 + q] = ok ? 0.1f : 0.0f;
        } else {
            t[3 + q] = 0.0f, w[3 + q] = fixed ? 0.0f : 0.01f;
        }
    }
}

__global__ void k_mlp_record_done(MlpDev M, int nf) { *M.scount += nf; }

// After the solve: each frame node's dv for the next substep's features
__global__ void k_mlp_store_dv(FemDev F, MlpDev M) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= F.nf) return;
    const int k = F.iperm[i];
    const bool fixed = F.fixed[k] != 0;
    for (int a = 0; a < 3; a++) M.prev_dv[3 * i + a] = fixed ? 0.0f : (float)F.rhs[6 * (size_t)k + a];
}

// ------------------------------------------------------------------------------------------ training
// The loss L = sum_s sum_o w_so (y_so - t_so)^2 / (2 n) over a batch of n samples (idx: the samples, null: x, t, w in
// order) and its gradient. A block strides over tiles of 32 samples: the forward, then layer by layer the weights'
// gradient (a thread a 4 x 4 patch of each matrix, its sums kept in registers over all the block's tiles) and the data
// gradient (a thread 2 samples x 4 inputs), in FP32 multiply-adds on rows in shared memory; at its end its share of the
// gradient (gpart: kParams a block) and loss (lpart). Every sum in a fixed order: deterministic.
// Reads of shared memory bound it (a multiply-add reads half a float of it; the arithmetic, 0.42 G multiply-adds at 20,660
// samples, is 12 us). B200, 20,660 samples: 477 us with a warp a block, a lane a sample and a share of the gradient stored
// a tile (29 MB), 72 us so; the sums over the blocks 48 and 10 us. Two blocks an SM: their tiles overlap each other's
// barriers.
struct MlpGradSmem {
    MlpTile T;
    float d[2][kTile * kPadF];  // the deltas of a layer's outputs and inputs
    float W[kHid * kHid * 2 + kOut * kHid]; // W2, W3, W4 as FP32
    double loss[kMlpThreads / 32];
};
// acc[o][i] += sum_s d[s][o0 + o] a[s][i0 + i]; db += sum_s d[s][ob]
__device__ __forceinline__ void mlp_outer(float (&acc)[4][4], const float* d, int ldd, const float* a, int o0, int i0) {
#pragma unroll 4
    for (int s = 0; s < kTile; s++) {
        const float4 dv = *reinterpret_cast<const float4*>(d + s * ldd + o0), av = *reinterpret_cast<const float4*>(a + s * kPadF + i0);
        const float dd[4] = {dv.x, dv.y, dv.z, dv.w}, aa[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
        for (int o = 0; o < 4; o++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[o][i] = fmaf(dd[o], aa[i], acc[o][i]);
    }
}
// din[s][i] = [act > 0] sum_o W[o][i] dout[s][o]: samples s0, s0 + 1, inputs i0 .. i0 + 3
template <int kN>
__device__ __forceinline__ void mlp_back(const float* W, const float* dout, int ldd, const float* act, float* din, int s0, int i0) {
    float r[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
#pragma unroll 4
    for (int o = 0; o < kN; o += 4) {
        const float4 d0 = *reinterpret_cast<const float4*>(dout + s0 * ldd + o), d1 = *reinterpret_cast<const float4*>(dout + (s0 + 1) * ldd + o);
        const float dd[2][4] = {{d0.x, d0.y, d0.z, d0.w}, {d1.x, d1.y, d1.z, d1.w}};
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float4 w = *reinterpret_cast<const float4*>(W + (o + u) * kHid + i0);
            const float ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int i = 0; i < 4; i++) r[q][i] = fmaf(ww[i], dd[q][u], r[q][i]);
        }
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const float4 a = *reinterpret_cast<const float4*>(act + (s0 + q) * kPadF + i0);
        *reinterpret_cast<float4*>(din + (s0 + q) * kPadF + i0) =
            make_float4(a.x > 0 ? r[q][0] : 0.0f, a.y > 0 ? r[q][1] : 0.0f, a.z > 0 ? r[q][2] : 0.0f, a.w > 0 ? r[q][3] : 0.0f);
    }
}

__global__ void __launch_bounds__(kMlpThreads, 2) k_mlp_grad(MlpDev M, const float* __restrict__ x, const float* __restrict__ t,
                                                             const float* __restrict__ w, const int* __restrict__ idx, int n, float* __restrict__ gpart,
                                                             double* __restrict__ lpart) {
    extern __shared__ __align__(16) unsigned char mlp_smem[];
    MlpGradSmem& S = *reinterpret_cast<MlpGradSmem*>(mlp_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    MlpFrag W;
    mlp_load(M.wb, W);
    float *W2 = S.W, *W3 = S.W + kHid * kHid, *W4 = S.W + 2 * kHid * kHid;
    for (int e = tid; e < kHid * kHid; e += kMlpThreads) W2[e] = __bfloat162float(M.wb[kOffW2 + e]), W3[e] = __bfloat162float(M.wb[kOffW3 + e]);
    for (int e = tid; e < kOut * kHid; e += kMlpThreads) W4[e] = __bfloat162float(M.wb[kOffW4 + e]);
    const int og = tid >> 4, ig = tid & 15, o0 = 4 * og, i0 = 4 * ig, s0 = 2 * og; // (this thread's patches)
    float g1[4][4], g2[4][4], g3[4][4], g4[4][4], b1 = 0, b2 = 0, b3 = 0, b4 = 0;
#pragma unroll
    for (int o = 0; o < 4; o++)
#pragma unroll
        for (int i = 0; i < 4; i++) g1[o][i] = g2[o][i] = g3[o][i] = g4[o][i] = 0.0f;
    auto bias = [&](float& b, const float* d, int ldd, int nout) {
        if (tid < nout)
            for (int s = 0; s < kTile; s++) b += d[s * ldd + tid];
    };
    double loss = 0.0;
    const float inv_n = 1.0f / (float)n;
    const int ntile = (n + kTile - 1) / kTile;
    for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const int q0 = tile * kTile;
        auto sample = [&](int smp) { return (size_t)(idx ? idx[q0 + smp] : q0 + smp); };
        mlp_forward(W, S.T, [&](int smp, int f) { return q0 + smp < n ? x[kIn * sample(smp) + f] : 0.0f; });
        // d4 = w (y - t) / n into y's place, its padding zero; the samples' loss
        for (int e = tid; e < kTile * 16; e += kMlpThreads) {
            const int smp = e >> 4, o = e & 15;
            float d = 0.0f;
            if (o < kOut && q0 + smp < n) {
                const size_t at = kOut * sample(smp) + o;
                const float wo = w[at], er = S.T.y[e] - t[at];
                loss += (double)(0.5f * wo * er * er);
                d = wo * er * inv_n;
            }
            S.T.y[e] = d;
        }
        __syncthreads();
        if (og < 3) mlp_outer(g4, S.T.y, 16, S.T.a[3], o0, i0);
        bias(b4, S.T.y, 16, kOut);
        mlp_back<kOut>(W4, S.T.y, 16, S.T.a[3], S.d[0], s0, i0);
        __syncthreads();
        mlp_outer(g3, S.d[0], kPadF, S.T.a[2], o0, i0);
        bias(b3, S.d[0], kPadF, kHid);
        mlp_back<kHid>(W3, S.d[0], kPadF, S.T.a[2], S.d[1], s0, i0);
        __syncthreads();
        mlp_outer(g2, S.d[1], kPadF, S.T.a[1], o0, i0);
        bias(b2, S.d[1], kPadF, kHid);
        mlp_back<kHid>(W2, S.d[1], kPadF, S.T.a[1], S.d[0], s0, i0);
        __syncthreads();
        if (ig < kIn / 4) mlp_outer(g1, S.d[0], kPadF, S.T.a[0], o0, i0);
        bias(b1, S.d[0], kPadF, kHid);
        __syncthreads();
    }
    float* g = gpart + (size_t)blockIdx.x * kParams;
#pragma unroll
    for (int o = 0; o < 4; o++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (ig < kIn / 4) g[kOffW1 + (o0 + o) * kIn + i0 + i] = g1[o][i];
            g[kOffW2 + (o0 + o) * kHid + i0 + i] = g2[o][i], g[kOffW3 + (o0 + o) * kHid + i0 + i] = g3[o][i];
            if (og < 3) g[kOffW4 + (o0 + o) * kHid + i0 + i] = g4[o][i];
        }
    if (tid < kHid) g[kOffB1 + tid] = b1, g[kOffB2 + tid] = b2, g[kOffB3 + tid] = b3;
    if (tid < kOut) g[kOffB4 + tid] = b4;
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0) S.loss[warp] = loss;
    __syncthreads();
    if (tid == 0) {
        double l = 0;
        for (int r = 0; r < kMlpThreads / 32; r++) l += S.loss[r];
        lpart[blockIdx.x] = l;
    }
}

// The blocks' gradients summed in a fixed order (into gsum; 8 groups of a block's threads each every 8th block's, then the
// groups in order), and, with lr > 0, one Adam step (t: its count from 1) of the FP32 parameters and their BF16 copy. The
// first block's second warp adds the blocks' losses to *acc.
__global__ void __launch_bounds__(256) k_mlp_adam(MlpDev M, const float* __restrict__ gpart, const double* __restrict__ lpart, int nblocks,
                                                  float* __restrict__ gsum, double* acc, float lr, float b1, float b2, float eps, int t) {
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5, p = blockIdx.x * 32 + lane;
    float g = 0.0f;
    if (p < kParams)
#pragma unroll 8
        for (int b = grp; b < nblocks; b += 8) g += gpart[(size_t)b * kParams + p];
    part[grp][lane] = g;
    __syncthreads();
    if (acc && blockIdx.x == 0 && grp == 1) {
        double s = 0;
        for (int b = lane; b < nblocks; b += 32) s += lpart[b];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) *acc += s;
    }
    if (grp != 0 || p >= kParams) return;
    g = 0.0f;
    for (int r = 0; r < 8; r++) g += part[r][lane];
    if (gsum) gsum[p] = g;
    if (!(lr > 0)) return;
    const float m = b1 * M.m[p] + (1.0f - b1) * g;
    const float v = b2 * M.v[p] + (1.0f - b2) * g * g;
    M.m[p] = m, M.v[p] = v;
    const float mh = m / (1.0f - powf(b1, (float)t)), vh = v / (1.0f - powf(b2, (float)t));
    const float wn = M.w[p] - lr * mh / (sqrtf(vh) + eps);
    M.w[p] = wn;
    ((__nv_bfloat16*)M.wb)[p] = __float2bfloat16(wn);
}

__global__ void k_mlp_sync_bf16(MlpDev M) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < kParams) ((__nv_bfloat16*)M.wb)[p] = __float2bfloat16(M.w[p]);
}

// The network's outputs for n samples
__global__ void __launch_bounds__(kMlpThreads) k_mlp_forward_batch(MlpDev M, const float* __restrict__ x, int n, float* __restrict__ y) {
    __shared__ __align__(16) MlpTile S;
    MlpFrag W;
    mlp_load(M.wb, W);
    for (int q0 = blockIdx.x * kTile; q0 < n; q0 += gridDim.x * kTile) {
        mlp_forward(W, S, [&](int smp, int f) { return q0 + smp < n ? x[(size_t)kIn * (q0 + smp) + f] : 0.0f; });
        for (int e = threadIdx.x; e < kTile * kOut; e += kMlpThreads)
            if (q0 + e / kOut < n) y[(size_t)kOut * q0 + e] = S.y[(e / kOut) * 16 + e % kOut];
        __syncthreads();
    }
}

} // namespace blg
