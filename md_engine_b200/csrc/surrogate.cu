// Learned surrogate of the E3B three-body forces (no reference counterpart;
// the exact term is ThreeBodyE3B.h:255-549 / EvaluatorE3B.h:145-345, which
// stays the fallback and the measure of the surrogate's force error).
//
// Model.  For molecule m a right-handed frame (e1 along the H-O-H bisector,
// e2 toward H1, e3 = e1 x e2) and 128 rotation-invariant features: four
// channels (O_m->O_j, O_m->H_j, H1_m->O_j, H2_m->O_j over the molecules j of
// the E3B molecule list), eight Gaussian radial shells per channel under a
// cosine cutoff of 5.6 A, and per shell the sum of the weights and of the
// weighted unit vectors in m's frame.  Standardised features go through an MLP
// 128 -> 64 -> 64 -> 64 -> 9 (SiLU) whose outputs are the three-body forces on
// O, H1 and H2 of m in m's frame (scaled by the training set's force RMS);
// they are rotated back to the lab frame.  Forces are not conservative (a
// regression surrogate, scored by force RMSE); the exact O-O two-body term is
// kept.
//
// Arithmetic.  Every GEMM uses BF16 operands with FP32 accumulation on the
// tensor cores (mma.sync m16n8k16 bf16): the inference kernel keeps the 64-wide
// activations in registers between layers; training runs forward, loss and
// backward of 64-row tiles in one kernel, then Adam on FP32 master weights.
#include <algorithm>
#include <cmath>
#include <random>
#include <vector>

#include <cstring>

#include "engine.hpp"

namespace mdx {

namespace {

using S = E3BSurrogate;
constexpr int kTeam = 8;      // lanes per molecule in the feature kernel
constexpr int kListTeam = kE3BTeam;  // team layout of the E3B molecule list
constexpr float kCut = 5.6f;  // feature cutoff (A)
constexpr float kPi = 3.14159265358979f;

// radial shells: channel 0 (O-O) centres 2.4 + 0.4 b, width 0.4; channels
// 1-3 (O-H, H-O) centres 1.5 + 0.5 b, width 0.5
__device__ __forceinline__ float shell_mu(int c, int b) { return c == 0 ? 2.4f + 0.4f * b : 1.5f + 0.5f * b; }
__device__ __forceinline__ float shell_gamma(int c) { return c == 0 ? 3.125f : 2.0f; }

struct FeatArgs {
    int nmol;
    const int4 *mol_idx;
    const float4 *xs;
    const uint32_t *mcounts, *mlist;
    int mcap;
    Box box;
    const float *mean, *inv_std;
    __nv_bfloat16 *feat;  // standardised BF16 [nmol_pad x kIn] (may be null)
    float *raw;           // raw FP32 [nmol x kIn] (may be null)
    float4 *frame;        // [3 nmol]: e1, e2, e3
};

__device__ __forceinline__ float3 nrm(float3 v) { return v * rsqrtf(dot3(v, v)); }

__device__ __forceinline__ void mol_frame(const float3 o, const float3 h1, const float3 h2, float3 &e1, float3 &e2,
                                          float3 &e3) {
    const float3 a = h1 - o, b = h2 - o;
    e1 = nrm(a + b);
    float3 d = a - b;
    d = d - e1 * dot3(d, e1);
    e2 = nrm(d);
    e3 = make_float3(e1.y * e2.z - e1.z * e2.y, e1.z * e2.x - e1.x * e2.z, e1.x * e2.y - e1.y * e2.x);
}

// lane t of the team: channel t / 2, shells 4 (t % 2) .. 4 (t % 2) + 3
__global__ void k_features(const FeatArgs A) {
    constexpr int G = 32 / kTeam;
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int a = lane / kTeam, t = lane % kTeam;
    const int m = warp * G + a;
    if (m >= A.nmol) return;  // team-uniform; no shuffles below
    const int ch = t >> 1, b0 = 4 * (t & 1);
    const int4 ix = A.mol_idx[m];
    const float3 o = f3(A.xs[ix.x]);
    const float3 h1 = o + min_image(A.box, f3(A.xs[ix.y]) - o);
    const float3 h2 = o + min_image(A.box, f3(A.xs[ix.z]) - o);
    float3 e1, e2, e3;
    mol_frame(o, h1, h2, e1, e2, e3);
    const float3 src = ch == 2 ? h1 : (ch == 3 ? h2 : o);
    float acc[4][4];
#pragma unroll
    for (int b = 0; b < 4; b++)
#pragma unroll
        for (int k = 0; k < 4; k++) acc[b][k] = 0.f;
    const float gam = shell_gamma(ch);
    float mu[4];
#pragma unroll
    for (int b = 0; b < 4; b++) mu[b] = shell_mu(ch, b0 + b);
    int cnt = (int)A.mcounts[m];
    cnt = cnt < A.mcap ? cnt : A.mcap;
    constexpr int GL = 32 / kListTeam;
    const uint32_t *row = A.mlist + (size_t)(m / GL) * A.mcap * GL + (m % GL) * kListTeam;
    for (int k = 0; k < cnt; k++) {
        const int mj = (int)row[(size_t)(k / kListTeam) * 32 + (k % kListTeam)];
        const int4 jx = A.mol_idx[mj];
        const int nv = ch == 1 ? 2 : 1;
        for (int v = 0; v < nv; v++) {
            const int tgt = ch == 1 ? (v == 0 ? jx.y : jx.z) : jx.x;
            const float3 d = min_image(A.box, f3(A.xs[tgt]) - src);
            const float r2 = dot3(d, d);
            if (r2 >= kCut * kCut || r2 < 1e-6f) continue;
            const float r = sqrtf(r2);
            const float ir = 1.0f / r;
            const float u1 = dot3(d, e1) * ir, u2 = dot3(d, e2) * ir, u3 = dot3(d, e3) * ir;
            const float fc = 0.5f * (cosf(kPi * r / kCut) + 1.0f);
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const float x = r - mu[b];
                const float g = expf(-gam * x * x) * fc;
                acc[b][0] += g;
                acc[b][1] += g * u1;
                acc[b][2] += g * u2;
                acc[b][3] += g * u3;
            }
        }
    }
    const int base = ch * 32 + b0 * 4;
#pragma unroll
    for (int b = 0; b < 4; b++)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int f = base + b * 4 + k;
            const float v = acc[b][k];
            if (A.raw) A.raw[(size_t)m * S::kIn + f] = v;
            if (A.feat) A.feat[(size_t)m * S::kIn + f] = __float2bfloat16((v - A.mean[f]) * A.inv_std[f]);
        }
    if (t == 0) {
        A.frame[3 * m] = make_float4(e1.x, e1.y, e1.z, 0.f);
        A.frame[3 * m + 1] = make_float4(e2.x, e2.y, e2.z, 0.f);
        A.frame[3 * m + 2] = make_float4(e3.x, e3.y, e3.z, 0.f);
    }
}

// exact three-body forces of O, H1, H2 rotated into the molecule frame
__global__ void k_targets(int nmol, const int4 *__restrict__ mol_idx, const float4 *__restrict__ frame,
                          const float4 *__restrict__ f, float *__restrict__ Y) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nmol) return;
    const int4 ix = mol_idx[m];
    const float3 e1 = f3(frame[3 * m]), e2 = f3(frame[3 * m + 1]), e3 = f3(frame[3 * m + 2]);
    const int at[3] = {ix.x, ix.y, ix.z};
    float *y = Y + (size_t)m * S::kOut;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float3 F = f3(f[at[k]]);
        y[3 * k] = dot3(F, e1);
        y[3 * k + 1] = dot3(F, e2);
        y[3 * k + 2] = dot3(F, e3);
    }
    for (int k = 9; k < S::kOut; k++) y[k] = 0.f;
}

// per-feature mean and 1/std over the dataset (FP64 sums); one block of 256 per feature
__global__ void k_stats(size_t n, const float *__restrict__ X, float *__restrict__ mean, float *__restrict__ inv_std) {
    __shared__ double s1[256], s2[256];
    const int f = blockIdx.x;
    double a = 0.0, b = 0.0;
    for (size_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = X[i * S::kIn + f];
        a += v;
        b += v * v;
    }
    s1[threadIdx.x] = a;
    s2[threadIdx.x] = b;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            s1[threadIdx.x] += s1[threadIdx.x + o];
            s2[threadIdx.x] += s2[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double mu = s1[0] / (double)n;
        const double var = s2[0] / (double)n - mu * mu;
        mean[f] = (float)mu;
        inv_std[f] = var > 1e-12 ? (float)(1.0 / sqrt(var)) : 1.0f;
    }
}

// sum of squares of the targets (FP64) for the force scale; blocks of 256
__global__ void k_target_ss(size_t n, const float *__restrict__ Y, double *out) {
    __shared__ double sh[256];
    double a = 0.0;
    for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n * 9; i += (size_t)gridDim.x * blockDim.x) {
        const double v = Y[(i / 9) * S::kOut + i % 9];
        a += v * v;
    }
    sh[threadIdx.x] = a;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(out, sh[0]);
}

// minibatch: row i of the batch is dataset row hash(seed, i) % n; features
// standardised to BF16, targets scaled
__global__ void k_gather_batch(int B, size_t n, uint64_t seed, const float *__restrict__ X, const float *__restrict__ Y,
                               const float *__restrict__ mean, const float *__restrict__ inv_std, float inv_scale,
                               __nv_bfloat16 *__restrict__ xb, float *__restrict__ yb) {
    const int i = blockIdx.x;
    uint64_t h = seed ^ (0x9E3779B97F4A7C15ull * (uint64_t)(i + 1));
    h ^= h >> 33;
    h *= 0xff51afd7ed558ccdull;
    h ^= h >> 33;
    h *= 0xc4ceb9fe1a85ec53ull;
    h ^= h >> 33;
    const size_t r = h % n;
    for (int f = threadIdx.x; f < S::kIn; f += blockDim.x)
        xb[(size_t)i * S::kIn + f] = __float2bfloat16((X[r * S::kIn + f] - mean[f]) * inv_std[f]);
    for (int k = threadIdx.x; k < S::kOut; k += blockDim.x)
        yb[(size_t)i * S::kOut + k] = k < 9 ? Y[r * S::kOut + k] * inv_scale : 0.f;
}

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

__device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], const uint32_t b[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z) {
    const float s = 1.0f / (1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// ---- training: forward, loss and backward of 64-row tiles in one kernel ---
// All operands of a tile live in shared memory as BF16 rows (padded by 8, so
// that the eight rows of an ldmatrix fall on distinct banks), weights included;
// pre-activations and the weight-gradient accumulators stay in registers (the
// warp that computes a 16 x 32 piece of a layer's output computes the same
// piece of its gradient), and a block writes its gradient out once.  As a chain of 25 GEMM, element-wise and column-sum launches that
// passed every activation through global memory, and summed the bias
// gradients with one thread per column, a call with 4,096 rows of host arrays
// took 789 us; it takes 248 us so, copies included.
constexpr int kTrainThreads = 256;
constexpr int kTileRows = 64;
constexpr int kPitchX = S::kIn + 8, kPitchH = S::kHid + 8, kPitchO = S::kOut + 8;

struct TrainShared {
    __nv_bfloat16 w1[S::kIn * kPitchH], w2[S::kHid * kPitchH], w3[S::kHid * kPitchH], w4[S::kHid * kPitchO];
    __nv_bfloat16 x[kTileRows * kPitchX];
    __nv_bfloat16 act[3][kTileRows * kPitchH];
    __nv_bfloat16 dz4[kTileRows * kPitchO], dz[2][kTileRows * kPitchH];
    float bias[3 * S::kHid + S::kOut];
    float db[kTileRows / 16][3 * S::kHid + S::kOut];  // bias gradients by row of warps
    double loss[kTrainThreads / 32];
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <bool TRANS>
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16 *p) {
    if (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(smem_addr(p)));
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(smem_addr(p)));
}
template <bool TRANS>
__device__ __forceinline__ void ldsm2(uint32_t (&r)[2], const __nv_bfloat16 *p) {
    if (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                     : "=r"(r[0]), "=r"(r[1])
                     : "r"(smem_addr(p)));
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
                     : "=r"(r[0]), "=r"(r[1])
                     : "r"(smem_addr(p)));
}

// acc[j] += A B for the 16 x 8 pieces (i0, n0 + 8 j), K deep.  A(i, k) at
// a[i pa + k], or a[k pa + i] (AT); B(k, n) at b[k pb + n], or b[n pb + k] (BN)
template <int K, int NT, bool AT, bool BN>
__device__ __forceinline__ void tile_mma(float (&acc)[NT][4], const __nv_bfloat16 *a, int pa, int i0,
                                         const __nv_bfloat16 *b, int pb, int n0, int lane) {
    const int r = lane & 7, q = lane >> 3;
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += 16) {
        uint32_t af[4];
        if (AT) ldsm4<true>(af, a + (k0 + r + (q & 2 ? 8 : 0)) * pa + i0 + (q & 1 ? 8 : 0));
        else ldsm4<false>(af, a + (i0 + (lane & 15)) * pa + k0 + (lane >> 4) * 8);
#pragma unroll
        for (int j = 0; j < NT; j++) {
            uint32_t bf[2];
            // (lanes 16..31 repeat the addresses of 0..15: x2 reads only those)
            if (BN) ldsm2<false>(bf, b + (n0 + 8 * j + r) * pb + k0 + (q & 1) * 8);
            else ldsm2<true>(bf, b + (k0 + r + (q & 1) * 8) * pb + n0 + 8 * j);
            mma_bf16(acc[j], af, bf);
        }
    }
}

__device__ __forceinline__ void store2(__nv_bfloat16 *p, float a, float b) {
    *reinterpret_cast<uint32_t *>(p) = pack2(__float2bfloat16(a), __float2bfloat16(b));
}

// this warp's 16 x 32 piece of a hidden layer's forward: z = in W + b, act = silu(z)
template <int K>
__device__ __forceinline__ void train_forward(float (&z)[4][4], const __nv_bfloat16 *in, int pin, const __nv_bfloat16 *w,
                                              const float *bias, __nv_bfloat16 *act, int i0, int n0, int lane) {
    const int gq = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int c = 0; c < 4; c++) z[j][c] = 0.f;
    tile_mma<K, 4, false, false>(z, in, pin, i0, w, kPitchH, n0, lane);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int col = n0 + 8 * j + 2 * tq;
#pragma unroll
        for (int c = 0; c < 4; c++) z[j][c] += bias[col + (c & 1)];
        store2(act + (i0 + gq) * kPitchH + col, silu(z[j][0]), silu(z[j][1]));
        store2(act + (i0 + gq + 8) * kPitchH + col, silu(z[j][2]), silu(z[j][3]));
    }
}

// the same piece of a hidden layer's gradient: dz = (dnext W^T) silu'(z), and
// the column sums of its BF16 values into db
template <int K>
__device__ __forceinline__ void train_backward(const float (&z)[4][4], const __nv_bfloat16 *dnext, int pd,
                                               const __nv_bfloat16 *w, int pw, __nv_bfloat16 *dz, float (&db)[4][2],
                                               int i0, int n0, int lane) {
    const int gq = lane >> 2, tq = lane & 3;
    float da[4][4];
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int c = 0; c < 4; c++) da[j][c] = 0.f;
    tile_mma<K, 4, false, true>(da, dnext, pd, i0, w, pw, n0, lane);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int col = n0 + 8 * j + 2 * tq;
        __nv_bfloat16 d[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            d[c] = __float2bfloat16(da[j][c] * dsilu(z[j][c]));
            db[j][c & 1] += __bfloat162float(d[c]);
        }
        *reinterpret_cast<uint32_t *>(dz + (i0 + gq) * kPitchH + col) = pack2(d[0], d[1]);
        *reinterpret_cast<uint32_t *>(dz + (i0 + gq + 8) * kPitchH + col) = pack2(d[2], d[3]);
    }
}

// a 16 x 8 piece of a weight gradient into the block's own
__device__ __forceinline__ void put_piece(float *g, int ld, int i0, int n0, const float (&acc)[4], int lane) {
    float *p = g + (size_t)(i0 + (lane >> 2)) * ld + n0 + 2 * (lane & 3);
    *reinterpret_cast<float2 *>(p) = make_float2(acc[0], acc[1]);
    *reinterpret_cast<float2 *>(p + 8 * ld) = make_float2(acc[2], acc[3]);
}
// column sums held by the four lanes of each column pair, over the warp's rows
template <int NT>
__device__ __forceinline__ void put_bias(float *b, int n0, const float (&db)[NT][2], int lane) {
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
            float v = db[j][c];
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane < 4) b[n0 + 8 * j + 2 * lane + c] = v;
        }
}

// B rows (a multiple of 64) of standardised BF16 features x and targets t:
// each block's gradient into its row of part, its sum of squared errors into
// part_loss (added up by k_sum_grad in a fixed order: with float atomics onto one
// gradient it would not repeat bit for bit)
__global__ void __launch_bounds__(kTrainThreads) k_fwd_bwd(int B, const __nv_bfloat16 *__restrict__ x,
                                                           const float *__restrict__ t,
                                                           const __nv_bfloat16 *__restrict__ wb,
                                                           const float *__restrict__ wf, float *__restrict__ part,
                                                           double *__restrict__ part_loss) {
    extern __shared__ __align__(16) char train_smem[];
    TrainShared &sh = *reinterpret_cast<TrainShared *>(train_smem);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int gq = lane >> 2, tq = lane & 3;
    const int wr = w & 3, wc = w >> 2;
    const int i0 = 16 * wr, n0 = 32 * wc;
    for (int i = tid; i < S::kIn * S::kHid; i += kTrainThreads)
        sh.w1[i / S::kHid * kPitchH + i % S::kHid] = wb[S::kOffW1 + i];
    for (int i = tid; i < S::kHid * S::kHid; i += kTrainThreads) {
        sh.w2[i / S::kHid * kPitchH + i % S::kHid] = wb[S::kOffW2 + i];
        sh.w3[i / S::kHid * kPitchH + i % S::kHid] = wb[S::kOffW3 + i];
    }
    for (int i = tid; i < S::kHid * S::kOut; i += kTrainThreads)
        sh.w4[i / S::kOut * kPitchO + i % S::kOut] = wb[S::kOffW4 + i];
    for (int i = tid; i < 3 * S::kHid + S::kOut; i += kTrainThreads) {
        const int l = i / S::kHid;
        sh.bias[i] = wf[(l == 0 ? S::kOffB1 : (l == 1 ? S::kOffB2 : (l == 2 ? S::kOffB3 : S::kOffB4))) + i - l * S::kHid];
    }
    // gradient pieces of this warp: dW1 rows i0 and i0 + 64, dW2 and dW3 rows
    // i0 (columns n0 .. n0 + 31), dW4 rows i0, columns 8 wc .. 8 wc + 7
    float g1[2][4][4] = {}, g2[4][4] = {}, g3[4][4] = {}, g4[1][4] = {};
    float b1[4][2] = {}, b2[4][2] = {}, b3[4][2] = {}, b4[1][2] = {};
    double lsum = 0.0;
    for (int row0 = blockIdx.x * kTileRows; row0 < B; row0 += gridDim.x * kTileRows) {
        __syncthreads();
        for (int i = tid; i < kTileRows * S::kIn / 8; i += kTrainThreads) {
            const int r = i / (S::kIn / 8), c = i % (S::kIn / 8);
            *reinterpret_cast<uint4 *>(sh.x + r * kPitchX + 8 * c) =
                *reinterpret_cast<const uint4 *>(x + (size_t)(row0 + r) * S::kIn + 8 * c);
        }
        __syncthreads();
        float z1[4][4], z2[4][4], z3[4][4];
        train_forward<S::kIn>(z1, sh.x, kPitchX, sh.w1, sh.bias, sh.act[0], i0, n0, lane);
        __syncthreads();
        train_forward<S::kHid>(z2, sh.act[0], kPitchH, sh.w2, sh.bias + S::kHid, sh.act[1], i0, n0, lane);
        __syncthreads();
        train_forward<S::kHid>(z3, sh.act[1], kPitchH, sh.w3, sh.bias + 2 * S::kHid, sh.act[2], i0, n0, lane);
        __syncthreads();
        {
            // outputs, the loss over the nine used ones and their gradient
            float y[1][4] = {};
            tile_mma<S::kHid, 1, false, false>(y, sh.act[2], kPitchH, i0, sh.w4, kPitchO, 8 * wc, lane);
            const int col = 8 * wc + 2 * tq;
            __nv_bfloat16 d[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int k = col + (c & 1), row = i0 + gq + (c & 2 ? 8 : 0);
                float g = 0.f;
                if (k < S::kOutUsed) {
                    const float e = y[0][c] + sh.bias[3 * S::kHid + k] - t[(size_t)(row0 + row) * S::kOut + k];
                    lsum += (double)e * e;
                    g = 2.0f * e / (float)(B * S::kOutUsed);
                }
                d[c] = __float2bfloat16(g);
                b4[0][c & 1] += __bfloat162float(d[c]);
            }
            *reinterpret_cast<uint32_t *>(sh.dz4 + (i0 + gq) * kPitchO + col) = pack2(d[0], d[1]);
            *reinterpret_cast<uint32_t *>(sh.dz4 + (i0 + gq + 8) * kPitchO + col) = pack2(d[2], d[3]);
        }
        __syncthreads();
        tile_mma<kTileRows, 1, true, false>(g4, sh.act[2], kPitchH, i0, sh.dz4, kPitchO, 8 * wc, lane);
        train_backward<S::kOut>(z3, sh.dz4, kPitchO, sh.w4, kPitchO, sh.dz[0], b3, i0, n0, lane);
        __syncthreads();
        tile_mma<kTileRows, 4, true, false>(g3, sh.act[1], kPitchH, i0, sh.dz[0], kPitchH, n0, lane);
        train_backward<S::kHid>(z2, sh.dz[0], kPitchH, sh.w3, kPitchH, sh.dz[1], b2, i0, n0, lane);
        __syncthreads();
        tile_mma<kTileRows, 4, true, false>(g2, sh.act[0], kPitchH, i0, sh.dz[1], kPitchH, n0, lane);
        train_backward<S::kHid>(z1, sh.dz[1], kPitchH, sh.w2, kPitchH, sh.dz[0], b1, i0, n0, lane);
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; h++)
            tile_mma<kTileRows, 4, true, false>(g1[h], sh.x, kPitchX, i0 + 64 * h, sh.dz[0], kPitchH, n0, lane);
    }
    float *const grad = part + (size_t)blockIdx.x * S::kParams;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        put_piece(grad + S::kOffW1, S::kHid, i0, n0 + 8 * j, g1[0][j], lane);
        put_piece(grad + S::kOffW1, S::kHid, i0 + 64, n0 + 8 * j, g1[1][j], lane);
        put_piece(grad + S::kOffW2, S::kHid, i0, n0 + 8 * j, g2[j], lane);
        put_piece(grad + S::kOffW3, S::kHid, i0, n0 + 8 * j, g3[j], lane);
    }
    put_piece(grad + S::kOffW4, S::kOut, i0, 8 * wc, g4[0], lane);
    put_bias(sh.db[wr], n0, b1, lane);
    put_bias(sh.db[wr] + S::kHid, n0, b2, lane);
    put_bias(sh.db[wr] + 2 * S::kHid, n0, b3, lane);
    put_bias(sh.db[wr] + 3 * S::kHid, 8 * wc, b4, lane);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if (lane == 0) sh.loss[w] = lsum;
    __syncthreads();
    for (int i = tid; i < 3 * S::kHid + S::kOut; i += kTrainThreads) {
        const int l = i / S::kHid;
        grad[(l == 0 ? S::kOffB1 : (l == 1 ? S::kOffB2 : (l == 2 ? S::kOffB3 : S::kOffB4))) + i - l * S::kHid] =
            (sh.db[0][i] + sh.db[1][i]) + (sh.db[2][i] + sh.db[3][i]);
    }
    if (tid == 0) {
        double l = 0.0;
        for (int k = 0; k < kTrainThreads / 32; k++) l += sh.loss[k];
        part_loss[blockIdx.x] = l;
    }
}

// the blocks' gradients and losses added up in a fixed order: four threads to
// a parameter, each a stretch of the rows (64 rows of 70 KB at 4,096 rows of a
// batch, read from L2)
constexpr int kSumCols = 64;
__global__ void __launch_bounds__(4 * kSumCols) k_sum_grad(int rows, const float *__restrict__ part,
                                                           const double *__restrict__ part_loss,
                                                           float *__restrict__ grad, double *__restrict__ loss) {
    __shared__ float sh[4][kSumCols];
    const int col = threadIdx.x % kSumCols, seg = threadIdx.x / kSumCols;
    const int i = blockIdx.x * kSumCols + col;
    const int per = (rows + 3) / 4, end = min(rows, (seg + 1) * per);
    float s = 0.f;
    if (i < S::kParams)
#pragma unroll 8
        for (int r = seg * per; r < end; r++) s += part[(size_t)r * S::kParams + i];
    sh[seg][col] = s;
    __syncthreads();
    if (seg == 0 && i < S::kParams) grad[i] = (sh[0][col] + sh[1][col]) + (sh[2][col] + sh[3][col]);
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        double l = 0.0;
        for (int r = threadIdx.x; r < rows; r += 32) l += part_loss[r];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (threadIdx.x == 0) *loss = l;
    }
}

__global__ void k_adam(int n, float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, float lr, float b1, float b2, float c1, float c2, float eps) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

__global__ void k_to_bf16(size_t n, const float *__restrict__ w, __nv_bfloat16 *__restrict__ wb) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) wb[i] = __float2bfloat16(w[i]);
}

// ---- inference: one warp per 16 molecules, weights in shared memory,
// activations kept in registers between layers (the m16n8k16 accumulator
// layout of two adjacent n-tiles is the A-operand layout of one k-tile)
struct InferArgs {
    int nmol;
    const __nv_bfloat16 *feat;  // [nmol_pad x kIn]
    const __nv_bfloat16 *wb;    // bf16 weights (blob offsets)
    const float *w;             // fp32 blob (biases)
    const float4 *frame;
    const int4 *mol_idx;
    float scale;
    float4 *out;  // forces: O gets +=, H1/H2 stored (side-buffer semantics)
    float *yraw;  // optional [nmol_pad x kOut] model outputs
    int add_o;
};

constexpr int kInferWarps = 4;

template <int KT, int NT>
__device__ __forceinline__ void layer(const uint32_t (&a)[KT][4], const __nv_bfloat16 *W, int ldw, const float *bias,
                                      float (&c)[NT][4], int lane) {
    const int gq = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const float b0 = bias[8 * j + 2 * tq], b1 = bias[8 * j + 2 * tq + 1];
        c[j][0] = b0;
        c[j][1] = b1;
        c[j][2] = b0;
        c[j][3] = b1;
    }
#pragma unroll
    for (int k = 0; k < KT; k++) {
#pragma unroll
        for (int j = 0; j < NT; j++) {
            const int kr = 16 * k + 2 * tq, nc = 8 * j + gq;
            uint32_t bf[2];
            bf[0] = pack2(W[kr * ldw + nc], W[(kr + 1) * ldw + nc]);
            bf[1] = pack2(W[(kr + 8) * ldw + nc], W[(kr + 9) * ldw + nc]);
            mma_bf16(c[j], a[k], bf);
        }
    }
}

template <int NT>
__device__ __forceinline__ void to_afrag(const float (&c)[NT][4], uint32_t (&a)[NT / 2][4]) {
#pragma unroll
    for (int k = 0; k < NT / 2; k++) {
        a[k][0] = pack2(__float2bfloat16(silu(c[2 * k][0])), __float2bfloat16(silu(c[2 * k][1])));
        a[k][1] = pack2(__float2bfloat16(silu(c[2 * k][2])), __float2bfloat16(silu(c[2 * k][3])));
        a[k][2] = pack2(__float2bfloat16(silu(c[2 * k + 1][0])), __float2bfloat16(silu(c[2 * k + 1][1])));
        a[k][3] = pack2(__float2bfloat16(silu(c[2 * k + 1][2])), __float2bfloat16(silu(c[2 * k + 1][3])));
    }
}

__global__ void __launch_bounds__(kInferWarps * 32) k_mlp_infer(const InferArgs A) {
    __shared__ __nv_bfloat16 sw[S::kOffB4];      // weights (bias slots unused)
    __shared__ float sb[3 * S::kHid + S::kOut];  // b1, b2, b3, b4
    __shared__ float sy[kInferWarps][16][S::kOut];
    for (int i = threadIdx.x; i < S::kOffB4; i += blockDim.x) sw[i] = A.wb[i];
    for (int i = threadIdx.x; i < 3 * S::kHid + S::kOut; i += blockDim.x) {
        const int l = i / S::kHid;
        const int off = l == 0 ? S::kOffB1 : (l == 1 ? S::kOffB2 : (l == 2 ? S::kOffB3 : S::kOffB4));
        sb[i] = A.w[off + i - l * S::kHid];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gq = lane >> 2, tq = lane & 3;
    const int r0 = (blockIdx.x * kInferWarps + w) * 16;
    if (r0 >= A.nmol) return;  // warp-uniform, after the only block barrier
    uint32_t x[8][4];
    const __nv_bfloat16 *F = A.feat + (size_t)r0 * S::kIn;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int c = 16 * k + 2 * tq;
        x[k][0] = pack2(F[gq * S::kIn + c], F[gq * S::kIn + c + 1]);
        x[k][1] = pack2(F[(gq + 8) * S::kIn + c], F[(gq + 8) * S::kIn + c + 1]);
        x[k][2] = pack2(F[gq * S::kIn + c + 8], F[gq * S::kIn + c + 9]);
        x[k][3] = pack2(F[(gq + 8) * S::kIn + c + 8], F[(gq + 8) * S::kIn + c + 9]);
    }
    float c1[8][4];
    layer<8, 8>(x, sw + S::kOffW1, S::kHid, sb, c1, lane);
    uint32_t a1[4][4];
    to_afrag<8>(c1, a1);
    float c2[8][4];
    layer<4, 8>(a1, sw + S::kOffW2, S::kHid, sb + S::kHid, c2, lane);
    uint32_t a2[4][4];
    to_afrag<8>(c2, a2);
    float c3[8][4];
    layer<4, 8>(a2, sw + S::kOffW3, S::kHid, sb + 2 * S::kHid, c3, lane);
    uint32_t a3[4][4];
    to_afrag<8>(c3, a3);
    float c4[2][4];
    layer<4, 2>(a3, sw + S::kOffW4, S::kOut, sb + 3 * S::kHid, c4, lane);
#pragma unroll
    for (int j = 0; j < 2; j++) {
        sy[w][gq][8 * j + 2 * tq] = c4[j][0];
        sy[w][gq][8 * j + 2 * tq + 1] = c4[j][1];
        sy[w][gq + 8][8 * j + 2 * tq] = c4[j][2];
        sy[w][gq + 8][8 * j + 2 * tq + 1] = c4[j][3];
    }
    __syncwarp();
    if (lane < 16) {
        const int m = r0 + lane;
        if (A.yraw)
            for (int k = 0; k < S::kOut; k++) A.yraw[(size_t)m * S::kOut + k] = sy[w][lane][k];
        if (m < A.nmol && A.out) {
            const float3 e1 = f3(A.frame[3 * m]), e2 = f3(A.frame[3 * m + 1]), e3 = f3(A.frame[3 * m + 2]);
            const int4 ix = A.mol_idx[m];
            const float *y = sy[w][lane];
            const float s = A.scale;
            const float3 fo = (e1 * y[0] + e2 * y[1] + e3 * y[2]) * s;
            const float3 fh1 = (e1 * y[3] + e2 * y[4] + e3 * y[5]) * s;
            const float3 fh2 = (e1 * y[6] + e2 * y[7] + e3 * y[8]) * s;
            float4 o = A.add_o ? A.out[ix.x] : make_float4(0.f, 0.f, 0.f, 0.f);
            A.out[ix.x] = make_float4(o.x + fo.x, o.y + fo.y, o.z + fo.z, 0.f);
            A.out[ix.y] = make_float4(fh1.x, fh1.y, fh1.z, 0.f);
            A.out[ix.z] = make_float4(fh2.x, fh2.y, fh2.z, 0.f);
        }
    }
}

__global__ void k_add_forces(int nmol, const int4 *__restrict__ mol_idx, const float4 *__restrict__ src,
                             float4 *__restrict__ fs) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nmol) return;
    const int4 ix = mol_idx[m];
    const int at[3] = {ix.x, ix.y, ix.z};
    for (int k = 0; k < 3; k++) {
        const float4 a = src[at[k]];
        float4 f = fs[at[k]];
        f.x += a.x;
        f.y += a.y;
        f.z += a.z;
        fs[at[k]] = f;
    }
}

// |surrogate - exact|^2 and |exact|^2 over O, H1, H2 of every molecule (FP64;
// blocks of 256)
__global__ void k_compare(int nmol, const int4 *__restrict__ mol_idx, const float4 *__restrict__ a,
                          const float4 *__restrict__ b, double *out) {
    __shared__ double s1[256], s2[256];
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    double d2 = 0.0, r2 = 0.0;
    if (m < nmol) {
        const int4 ix = mol_idx[m];
        const int at[3] = {ix.x, ix.y, ix.z};
        for (int k = 0; k < 3; k++) {
            const float4 x = a[at[k]], y = b[at[k]];
            const double dx = x.x - y.x, dy = x.y - y.y, dz = x.z - y.z;
            d2 += dx * dx + dy * dy + dz * dz;
            r2 += (double)y.x * y.x + (double)y.y * y.y + (double)y.z * y.z;
        }
    }
    s1[threadIdx.x] = d2;
    s2[threadIdx.x] = r2;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            s1[threadIdx.x] += s1[threadIdx.x + o];
            s2[threadIdx.x] += s2[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        atomicAdd(out, s1[0]);
        atomicAdd(out + 1, s2[0]);
    }
}

int pad16(int n) { return (n + 15) / 16 * 16; }

int sur_alloc(State &s, FixE3B &f) {
    if (!f.sur) f.sur.reset(new E3BSurrogate());
    S &u = *f.sur;
    const int nmol = (int)f.mol_ids.size();
    const int np = pad16(std::max(nmol, 1)) + 64;  // + a block of padding rows
    if (int e = u.feat.alloc((size_t)np * S::kIn)) return e;
    if (int e = u.raw.alloc((size_t)std::max(nmol, 1) * S::kIn)) return e;
    if (int e = u.frame.alloc(3 * (size_t)std::max(nmol, 1))) return e;
    if (int e = u.fexact.alloc(std::max(s.gpd.n, 1))) return e;
    if (!u.w.p) {
        if (int e = u.w.alloc(S::kParams)) return e;
        if (int e = u.wb.alloc(S::kParams)) return e;
        if (int e = u.grad.alloc(S::kParams)) return e;
        if (int e = u.adam_m.alloc(S::kParams)) return e;
        if (int e = u.adam_v.alloc(S::kParams)) return e;
        if (int e = u.mean.alloc(S::kIn)) return e;
        if (int e = u.inv_std.alloc(S::kIn)) return e;
        if (int e = u.loss.alloc(1)) return e;
        // He-uniform weights (output layer x 0.1), zero biases, seeded
        std::vector<float> h(S::kParams, 0.f);
        std::mt19937_64 rng(20261203);
        auto fill = [&](int off, int fan_in, int count, float gain) {
            const float lim = gain * std::sqrt(6.0f / (float)fan_in);
            std::uniform_real_distribution<float> U(-lim, lim);
            for (int i = 0; i < count; i++) h[off + i] = U(rng);
        };
        fill(S::kOffW1, S::kIn, S::kIn * S::kHid, 1.0f);
        fill(S::kOffW2, S::kHid, S::kHid * S::kHid, 1.0f);
        fill(S::kOffW3, S::kHid, S::kHid * S::kHid, 1.0f);
        fill(S::kOffW4, S::kHid, S::kHid * S::kOut, 0.1f);
        for (int j = 0; j < S::kHid; j++)
            for (int k = S::kOutUsed; k < S::kOut; k++) h[S::kOffW4 + j * S::kOut + k] = 0.f;
        MDX_CUDA_TRY(cudaMemcpy(u.w.p, h.data(), S::kParams * sizeof(float), cudaMemcpyHostToDevice));
        MDX_CUDA_TRY(cudaMemset(u.adam_m.p, 0, S::kParams * sizeof(float)));
        MDX_CUDA_TRY(cudaMemset(u.adam_v.p, 0, S::kParams * sizeof(float)));
        std::vector<float> z(S::kIn, 0.f), o(S::kIn, 1.f);
        MDX_CUDA_TRY(cudaMemcpy(u.mean.p, z.data(), S::kIn * sizeof(float), cudaMemcpyHostToDevice));
        MDX_CUDA_TRY(cudaMemcpy(u.inv_std.p, o.data(), S::kIn * sizeof(float), cudaMemcpyHostToDevice));
        k_to_bf16<<<(S::kParams + 255) / 256, 256, 0, s.stream>>>(S::kParams, u.w.p, u.wb.p);
        MDX_LAUNCHED();
    }
    return 0;
}

FeatArgs feat_args(State &s, FixE3B &f) {
    S &u = *f.sur;
    FeatArgs A{};
    A.nmol = (int)f.mol_ids.size();
    A.mol_idx = f.d_mol_idx.p;
    A.xs = s.gpd.xs.p;
    A.mcounts = f.mcounts.p;
    A.mlist = f.mlist.p;
    A.mcap = f.mcap;
    A.box = s.box;
    A.mean = u.mean.p;
    A.inv_std = u.inv_std.p;
    A.feat = u.feat.p;
    A.raw = nullptr;
    A.frame = u.frame.p;
    return A;
}

dim3 feat_blocks(int nmol) {
    const int warps = (nmol + (32 / kTeam) - 1) / (32 / kTeam);
    return dim3((warps * 32 + 255) / 256);
}

InferArgs infer_args(FixE3B &f, int nmol, float4 *out, int add_o) {
    S &u = *f.sur;
    InferArgs I{};
    I.nmol = nmol;
    I.feat = u.feat.p;
    I.wb = u.wb.p;
    I.w = u.w.p;
    I.frame = u.frame.p;
    I.mol_idx = f.d_mol_idx.p;
    I.scale = u.force_scale;
    I.out = out;
    I.yraw = nullptr;
    I.add_o = add_o;
    return I;
}

unsigned infer_blocks(int n) { return (unsigned)((pad16(n) / 16 + kInferWarps - 1) / kInferWarps); }

// forward + backward of one minibatch already in u.xb / u.yb (B rows);
// gradient into u.grad, loss sum into u.loss
int sur_blocks(int B) { return std::min(B / kTileRows, num_sms()); }
int sur_fwd_bwd(S &u, int B, cudaStream_t st) {
    if (B % kTileRows) {
        set_error(MDX_ERR_ARG, "surrogate batch of %d rows not tiled by %d", B, kTileRows);
        return MDX_ERR_ARG;
    }
    MDX_CUDA_TRY(cudaFuncSetAttribute(k_fwd_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainShared)));
    const int nb = sur_blocks(B);
    k_fwd_bwd<<<nb, kTrainThreads, sizeof(TrainShared), st>>>(B, u.xb.p, u.yb.p, u.wb.p, u.w.p, u.part.p,
                                                              u.part_loss.p);
    MDX_LAUNCHED();
    k_sum_grad<<<(S::kParams + kSumCols - 1) / kSumCols, 4 * kSumCols, 0, st>>>(nb, u.part.p, u.part_loss.p, u.grad.p,
                                                                               u.loss.p);
    MDX_LAUNCHED();
    MDX_CUDA_TRY(cudaGetLastError());
    return 0;
}

int sur_batch_alloc(S &u, int B) {
    if (u.batch >= B) return 0;
    if (int e = u.xb.alloc((size_t)B * S::kIn)) return e;
    if (int e = u.yb.alloc((size_t)B * S::kOut)) return e;
    if (int e = u.part.alloc(std::max((size_t)sur_blocks(B) * S::kParams, (size_t)B * S::kIn))) return e;
    if (int e = u.part_loss.alloc(sur_blocks(B))) return e;
    u.batch = B;
    return 0;
}

FixE3B *e3b_of(mdx_fix *f) {
    if (!f || !f->f || f->f->kind != FixKind::E3B) return nullptr;
    return static_cast<FixE3B *>(f->f);
}

}  // namespace

// the surrogate's E3B forces of one step into the side buffer: exact two-body
// on O (stored), surrogate three-body added on O and stored on H1, H2
int surrogate_forces_to(State &s, FixE3B &f, float4 *out, cudaStream_t stream) {
    const int nmol = (int)f.mol_ids.size();
    if (nmol == 0) return 0;
    if (int e = e3b_twobody_to(s, f, out, stream)) return e;
    k_features<<<feat_blocks(nmol), 256, 0, stream>>>(feat_args(s, f));
    MDX_LAUNCHED();
    k_mlp_infer<<<infer_blocks(nmol), kInferWarps * 32, 0, stream>>>(infer_args(f, nmol, out, 1));
    MDX_LAUNCHED();
    return 0;
}

// FixE3B::compute with the surrogate on: the step's E3B forces added to fs
int surrogate_compute(State &s, FixE3B &f) {
    S &u = *f.sur;
    if (int e = surrogate_forces_to(s, f, u.fexact.p, s.stream)) return e;
    const int nmol = (int)f.mol_ids.size();
    k_add_forces<<<(nmol + 127) / 128, 128, 0, s.stream>>>(nmol, f.d_mol_idx.p, u.fexact.p, s.gpd.fs.p);
    MDX_LAUNCHED();
    return 0;
}

}  // namespace mdx

using namespace mdx;

static int need_prepared(mdx_state *st, FixE3B *f) {
    if (!st || !f) {
        set_error(MDX_ERR_ARG, "need a state and an E3B fix");
        return MDX_ERR_ARG;
    }
    if (!st->s->prepared || !f->prepared) {
        set_error(MDX_ERR_STATE, "call mdx_prepare first");
        return MDX_ERR_STATE;
    }
    return 0;
}

extern "C" {

// append the current frame (features + exact three-body forces in the molecule frames)
int mdx_e3b_surrogate_collect(mdx_state *st, mdx_fix *fix) {
    FixE3B *f = e3b_of(fix);
    if (int e = need_prepared(st, f)) return e;
    State &s = *st->s;
    if (int e = sur_alloc(s, *f)) return e;
    S &u = *f->sur;
    const int nmol = (int)f->mol_ids.size();
    if (u.n + nmol > u.cap) {
        size_t nc = std::max(u.cap * 2, u.n + nmol);
        nc = std::max(nc, (size_t)nmol * 16);
        DBuf<float> X2, Y2;
        if (int e = X2.alloc(nc * S::kIn)) return e;
        if (int e = Y2.alloc(nc * S::kOut)) return e;
        if (u.n) {
            MDX_CUDA_TRY(cudaMemcpyAsync(X2.p, u.X.p, u.n * S::kIn * sizeof(float), cudaMemcpyDeviceToDevice,
                                         s.stream));
            MDX_CUDA_TRY(cudaMemcpyAsync(Y2.p, u.Y.p, u.n * S::kOut * sizeof(float), cudaMemcpyDeviceToDevice,
                                         s.stream));
        }
        MDX_CUDA_TRY(cudaStreamSynchronize(s.stream));
        std::swap(u.X.p, X2.p);
        std::swap(u.X.n, X2.n);
        std::swap(u.Y.p, Y2.p);
        std::swap(u.Y.n, Y2.n);
        u.cap = nc;
    }
    if (int e = e3b_exact_to(s, *f, u.fexact.p, 0, s.stream)) return e;
    FeatArgs A = feat_args(s, *f);
    A.feat = nullptr;
    A.raw = u.X.p + u.n * S::kIn;
    k_features<<<feat_blocks(nmol), 256, 0, s.stream>>>(A);
    MDX_LAUNCHED();
    k_targets<<<(nmol + 127) / 128, 128, 0, s.stream>>>(nmol, f->d_mol_idx.p, u.frame.p, u.fexact.p,
                                                        u.Y.p + u.n * S::kOut);
    MDX_LAUNCHED();
    MDX_CUDA_TRY(cudaStreamSynchronize(s.stream));
    MDX_CUDA_TRY(cudaGetLastError());
    u.n += nmol;
    return 0;
}

int mdx_e3b_surrogate_dataset_size(mdx_fix *fix, int64_t *n) {
    FixE3B *f = e3b_of(fix);
    if (!f || !n) {
        set_error(MDX_ERR_ARG, "need an E3B fix");
        return MDX_ERR_ARG;
    }
    *n = f->sur ? (int64_t)f->sur->n : 0;
    return 0;
}

// standardisation statistics and force scale from the collected frames (first
// call), then `iters` Adam steps on minibatches of `batch` rows
int mdx_e3b_surrogate_train(mdx_state *st, mdx_fix *fix, int iters, int batch, float lr, uint64_t seed,
                            double *loss_first, double *loss_last) {
    FixE3B *f = e3b_of(fix);
    if (int e = need_prepared(st, f)) return e;
    State &s = *st->s;
    if (!f->sur || f->sur->n < 64) {
        set_error(MDX_ERR_STATE, "collect frames first (mdx_e3b_surrogate_collect)");
        return MDX_ERR_STATE;
    }
    if (iters < 0 || batch < 64 || batch % 64) {
        set_error(MDX_ERR_ARG, "batch must be a positive multiple of 64");
        return MDX_ERR_ARG;
    }
    S &u = *f->sur;
    cudaStream_t cs = s.stream;
    if (!u.stats) {
        k_stats<<<S::kIn, 256, 0, cs>>>(u.n, u.X.p, u.mean.p, u.inv_std.p);
        MDX_LAUNCHED();
        MDX_CUDA_TRY(cudaMemsetAsync(u.loss.p, 0, sizeof(double), cs));
        k_target_ss<<<148, 256, 0, cs>>>(u.n, u.Y.p, u.loss.p);
        MDX_LAUNCHED();
        double ss = 0.0;
        MDX_CUDA_TRY(cudaMemcpyAsync(&ss, u.loss.p, sizeof(double), cudaMemcpyDeviceToHost, cs));
        MDX_CUDA_TRY(cudaStreamSynchronize(cs));
        u.force_scale = (float)std::sqrt(ss / (double)(u.n * 9));
        if (!(u.force_scale > 0.f)) u.force_scale = 1.f;
        u.stats = true;
    }
    if (int e = sur_batch_alloc(u, batch)) return e;
    double lf = -1, ll = -1;
    for (int it = 0; it < iters; it++) {
        k_gather_batch<<<batch, 128, 0, cs>>>(batch, u.n, seed + 0x632BE59BD9B4E019ull * (uint64_t)(u.adam_t + 1),
                                              u.X.p, u.Y.p, u.mean.p, u.inv_std.p, 1.0f / u.force_scale, u.xb.p,
                                              u.yb.p);
        MDX_LAUNCHED();
        if (int e = sur_fwd_bwd(u, batch, cs)) return e;
        u.adam_t += 1;
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.f - std::pow(b1, (float)u.adam_t), c2 = 1.f - std::pow(b2, (float)u.adam_t);
        k_adam<<<(S::kParams + 255) / 256, 256, 0, cs>>>(S::kParams, u.w.p, u.grad.p, u.adam_m.p, u.adam_v.p, lr, b1,
                                                        b2, c1, c2, 1e-8f);
        MDX_LAUNCHED();
        k_to_bf16<<<(S::kParams + 255) / 256, 256, 0, cs>>>(S::kParams, u.w.p, u.wb.p);
        MDX_LAUNCHED();
        if (it == 0 || it == iters - 1) {
            double l = 0.0;
            MDX_CUDA_TRY(cudaMemcpyAsync(&l, u.loss.p, sizeof(double), cudaMemcpyDeviceToHost, cs));
            MDX_CUDA_TRY(cudaStreamSynchronize(cs));
            l /= (double)batch * 9.0;
            if (it == 0) lf = l;
            ll = l;
        }
    }
    MDX_CUDA_TRY(cudaStreamSynchronize(cs));
    MDX_CUDA_TRY(cudaGetLastError());
    u.trained = true;
    if (loss_first) *loss_first = lf;
    if (loss_last) *loss_last = ll;
    return 0;
}

// surrogate on (1) / exact E3B (0) for the fix's force evaluations
int mdx_e3b_surrogate_enable(mdx_fix *fix, int on) {
    FixE3B *f = e3b_of(fix);
    if (!f) {
        set_error(MDX_ERR_ARG, "need an E3B fix");
        return MDX_ERR_ARG;
    }
    if (on && (!f->sur || !f->sur->trained)) {
        set_error(MDX_ERR_STATE, "the surrogate is not trained");
        return MDX_ERR_STATE;
    }
    if (f->sur) f->sur->enabled = on != 0;
    return 0;
}

// three-body force error of the surrogate on the current frame:
// rmse = sqrt(mean |F_sur - F_exact|^2), rms = sqrt(mean |F_exact|^2) over O, H1, H2
int mdx_e3b_surrogate_eval(mdx_state *st, mdx_fix *fix, double *rmse, double *rms) {
    FixE3B *f = e3b_of(fix);
    if (int e = need_prepared(st, f)) return e;
    if (!f->sur || !f->sur->trained) {
        set_error(MDX_ERR_STATE, "the surrogate is not trained");
        return MDX_ERR_STATE;
    }
    State &s = *st->s;
    S &u = *f->sur;
    const int nmol = (int)f->mol_ids.size();
    DBuf<float4> fs;
    DBuf<double> acc;
    if (int e = fs.alloc(s.gpd.n)) return e;
    if (int e = acc.alloc(2)) return e;
    MDX_CUDA_TRY(cudaMemsetAsync(fs.p, 0, s.gpd.n * sizeof(float4), s.stream));
    MDX_CUDA_TRY(cudaMemsetAsync(acc.p, 0, 2 * sizeof(double), s.stream));
    if (int e = e3b_exact_to(s, *f, u.fexact.p, 0, s.stream)) return e;
    k_features<<<feat_blocks(nmol), 256, 0, s.stream>>>(feat_args(s, *f));
    MDX_LAUNCHED();
    k_mlp_infer<<<infer_blocks(nmol), kInferWarps * 32, 0, s.stream>>>(infer_args(*f, nmol, fs.p, 0));
    MDX_LAUNCHED();
    k_compare<<<(nmol + 255) / 256, 256, 0, s.stream>>>(nmol, f->d_mol_idx.p, fs.p, u.fexact.p, acc.p);
    MDX_LAUNCHED();
    double h[2];
    MDX_CUDA_TRY(cudaMemcpyAsync(h, acc.p, sizeof(h), cudaMemcpyDeviceToHost, s.stream));
    MDX_CUDA_TRY(cudaStreamSynchronize(s.stream));
    const double cnt = 3.0 * nmol;
    if (rmse) *rmse = std::sqrt(h[0] / cnt);
    if (rms) *rms = std::sqrt(h[1] / cnt);
    return 0;
}

// parameters: w (kParams floats), mean / inv_std (kIn floats), scale; any may be NULL
int mdx_e3b_surrogate_get_params(mdx_fix *fix, float *w, float *mean, float *inv_std, float *scale) {
    FixE3B *f = e3b_of(fix);
    if (!f || !f->sur || !f->sur->w.p) {
        set_error(MDX_ERR_STATE, "no surrogate on this fix (collect or set parameters first)");
        return MDX_ERR_STATE;
    }
    S &u = *f->sur;
    if (w) MDX_CUDA_TRY(cudaMemcpy(w, u.w.p, S::kParams * sizeof(float), cudaMemcpyDeviceToHost));
    if (mean) MDX_CUDA_TRY(cudaMemcpy(mean, u.mean.p, S::kIn * sizeof(float), cudaMemcpyDeviceToHost));
    if (inv_std) MDX_CUDA_TRY(cudaMemcpy(inv_std, u.inv_std.p, S::kIn * sizeof(float), cudaMemcpyDeviceToHost));
    if (scale) *scale = u.force_scale;
    return 0;
}

int mdx_e3b_surrogate_set_params(mdx_state *st, mdx_fix *fix, const float *w, const float *mean, const float *inv_std,
                                 float scale) {
    FixE3B *f = e3b_of(fix);
    if (int e = need_prepared(st, f)) return e;
    if (!w || !mean || !inv_std || !(scale > 0.f)) {
        set_error(MDX_ERR_ARG, "need weights, statistics and a positive scale");
        return MDX_ERR_ARG;
    }
    State &s = *st->s;
    if (int e = sur_alloc(s, *f)) return e;
    S &u = *f->sur;
    MDX_CUDA_TRY(cudaMemcpy(u.w.p, w, S::kParams * sizeof(float), cudaMemcpyHostToDevice));
    MDX_CUDA_TRY(cudaMemcpy(u.mean.p, mean, S::kIn * sizeof(float), cudaMemcpyHostToDevice));
    MDX_CUDA_TRY(cudaMemcpy(u.inv_std.p, inv_std, S::kIn * sizeof(float), cudaMemcpyHostToDevice));
    k_to_bf16<<<(S::kParams + 255) / 256, 256, 0, s.stream>>>(S::kParams, u.w.p, u.wb.p);
    MDX_LAUNCHED();
    MDX_CUDA_TRY(cudaStreamSynchronize(s.stream));
    u.force_scale = scale;
    u.stats = true;
    u.trained = true;
    return 0;
}

// raw features (nmol x kIn, FP32, molecule order of the fix) and frames
// (nmol x 9: e1, e2, e3) of the current positions
int mdx_e3b_surrogate_features(mdx_state *st, mdx_fix *fix, float *raw, float *frames) {
    FixE3B *f = e3b_of(fix);
    if (int e = need_prepared(st, f)) return e;
    State &s = *st->s;
    if (int e = sur_alloc(s, *f)) return e;
    S &u = *f->sur;
    const int nmol = (int)f->mol_ids.size();
    FeatArgs A = feat_args(s, *f);
    A.feat = nullptr;
    A.raw = u.raw.p;
    k_features<<<feat_blocks(nmol), 256, 0, s.stream>>>(A);
    MDX_LAUNCHED();
    MDX_CUDA_TRY(cudaStreamSynchronize(s.stream));
    // rows come per E3B molecule index; in the molecule form that index is the
    // slot, mapped back here to the fix's molecule order (FixRigid's maps)
    std::vector<int> row_of(nmol);
    for (int m = 0; m < nmol; m++) row_of[m] = m;
    if (s.mf.on) {
        std::vector<int4> mi(nmol);
        MDX_CUDA_TRY(cudaMemcpy(mi.data(), s.rigidFix()->d_mol_idx.p, nmol * sizeof(int4), cudaMemcpyDeviceToHost));
        for (int m = 0; m < nmol; m++) row_of[m] = mi[m].x >> 2;
    }
    if (raw) {
        std::vector<float> h((size_t)nmol * S::kIn);
        MDX_CUDA_TRY(cudaMemcpy(h.data(), u.raw.p, h.size() * sizeof(float), cudaMemcpyDeviceToHost));
        for (int m = 0; m < nmol; m++)
            std::memcpy(raw + (size_t)m * S::kIn, h.data() + (size_t)row_of[m] * S::kIn, S::kIn * sizeof(float));
    }
    if (frames) {
        std::vector<float4> h(3 * (size_t)nmol);
        MDX_CUDA_TRY(cudaMemcpy(h.data(), u.frame.p, h.size() * sizeof(float4), cudaMemcpyDeviceToHost));
        for (int m = 0; m < nmol; m++)
            for (int c = 0; c < 3; c++) {
                const float4 v = h[3 * (size_t)row_of[m] + c];
                frames[9 * (size_t)m + 3 * c] = v.x;
                frames[9 * (size_t)m + 3 * c + 1] = v.y;
                frames[9 * (size_t)m + 3 * c + 2] = v.z;
            }
    }
    return 0;
}

// model outputs for n standardised feature rows given on the host (rounded to
// BF16 on upload): y (n x kOut)
int mdx_e3b_surrogate_infer(mdx_state *st, mdx_fix *fix, const float *x, int n, float *y) {
    FixE3B *f = e3b_of(fix);
    if (int e = need_prepared(st, f)) return e;
    if (!f->sur || !x || !y || n <= 0) {
        set_error(MDX_ERR_ARG, "need a surrogate, inputs and outputs");
        return MDX_ERR_ARG;
    }
    State &s = *st->s;
    S &u = *f->sur;
    const int np = pad16(n) + 64;
    DBuf<__nv_bfloat16> xd;
    DBuf<float> yd;
    if (int e = xd.alloc((size_t)np * S::kIn)) return e;
    if (int e = yd.alloc((size_t)np * S::kOut)) return e;
    // rounded to BF16 on the device; the padding rows are zero
    const size_t nx = (size_t)n * S::kIn;
    if (int e = u.xf.alloc(nx)) return e;
    MDX_CUDA_TRY(cudaMemcpyAsync(u.xf.p, x, nx * sizeof(float), cudaMemcpyHostToDevice, s.stream));
    MDX_CUDA_TRY(cudaMemsetAsync(xd.p + nx, 0, ((size_t)np * S::kIn - nx) * sizeof(__nv_bfloat16), s.stream));
    k_to_bf16<<<(unsigned)((nx + 255) / 256), 256, 0, s.stream>>>(nx, u.xf.p, xd.p);
    MDX_LAUNCHED();
    InferArgs I = infer_args(*f, n, nullptr, 0);
    I.feat = xd.p;
    I.yraw = yd.p;
    I.w = u.w.p;
    k_mlp_infer<<<infer_blocks(n), kInferWarps * 32, 0, s.stream>>>(I);
    MDX_LAUNCHED();
    MDX_CUDA_TRY(cudaStreamSynchronize(s.stream));
    MDX_CUDA_TRY(cudaMemcpy(y, yd.p, (size_t)n * S::kOut * sizeof(float), cudaMemcpyDeviceToHost));
    return 0;
}

// loss (mean over n x 9) and gradient (kParams floats) of one minibatch given
// on the host: x standardised features (n x kIn), t scaled targets (n x kOut);
// n a multiple of 64.  No parameter update.
int mdx_e3b_surrogate_grad(mdx_state *st, mdx_fix *fix, const float *x, const float *t, int n, float *grad,
                           double *loss) {
    FixE3B *f = e3b_of(fix);
    if (int e = need_prepared(st, f)) return e;
    if (!f->sur || !x || !t || n <= 0 || n % 64) {
        set_error(MDX_ERR_ARG, "need a surrogate and n a positive multiple of 64");
        return MDX_ERR_ARG;
    }
    State &s = *st->s;
    S &u = *f->sur;
    if (int e = sur_batch_alloc(u, n)) return e;
    // rounded to BF16 on the device
    MDX_CUDA_TRY(cudaMemcpyAsync(u.part.p, x, (size_t)n * S::kIn * sizeof(float), cudaMemcpyHostToDevice, s.stream));
    k_to_bf16<<<(unsigned)(((size_t)n * S::kIn + 255) / 256), 256, 0, s.stream>>>((size_t)n * S::kIn, u.part.p, u.xb.p);
    MDX_LAUNCHED();
    MDX_CUDA_TRY(cudaMemcpyAsync(u.yb.p, t, (size_t)n * S::kOut * sizeof(float), cudaMemcpyHostToDevice, s.stream));
    if (int e = sur_fwd_bwd(u, n, s.stream)) return e;
    double l = 0.0;
    MDX_CUDA_TRY(cudaMemcpyAsync(&l, u.loss.p, sizeof(double), cudaMemcpyDeviceToHost, s.stream));
    MDX_CUDA_TRY(cudaStreamSynchronize(s.stream));
    if (grad) MDX_CUDA_TRY(cudaMemcpy(grad, u.grad.p, S::kParams * sizeof(float), cudaMemcpyDeviceToHost));
    if (loss) *loss = l / ((double)n * 9.0);
    return 0;
}

}  // extern "C"
