// P3M reciprocal-space Ewald (FixChargeEwald, src/Fixes/FixChargeEwald.cu).
//
//  spread   map_charge_to_grid_order_5_cu (:174-217): order-5 charge
//           assignment W_p_5 (:163-172), float atomics into a REAL grid
//  FFT      own transforms on cubic 32^3, 64^3 and 128^3 meshes (below); on
//           others cuFFT R2C (the reference runs C2C on a complex grid with a zero
//           imaginary part, :1307-1309; R2C computes the same half spectrum)
//  E(k)     E_field_cu (:386-434): E_d(k) = i k_d G(k) rho(k).  The reference
//           keeps only the real part after its C2C inverse, which drops the
//           anti-Hermitian Nyquist-plane term of each component; that term is
//           zeroed here so the C2R inverse gives the identical real field.
//  inverse  as the FFT; on other meshes one batched cuFFT C2R for the three
//           components (:1340-1346)
//  gather   Ewald_long_range_forces_order_5_cu (:561-630): F = Q q sum W E,
//           E = -ifft / V
//  G(k)     Green_function_cu (:314-366), evaluated once per box in FP64.
//  alpha    find_optimal_parameters (:848-967), secant on the RMS errors.
//
// Deviation (documented): the reference's nearest grid point is
// make_int3((x-lo+h/2)/h), a truncation toward zero, which mis-assigns the
// stencil of an atom more than h/2 below lo (atoms drift out of the box
// between list rebuilds); floorf is used here.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "engine.hpp"

namespace mdx {

namespace {

__device__ __forceinline__ void w5(float x, float w[5]) {
    const float x2 = x * x, x4 = x2 * x2;
    w[0] = (1.0f / 384.0f) * (1.0f - 8.0f * x + 24.0f * x2 - 32.0f * x * x2 + 16.0f * x4);
    w[1] = (1.0f / 96.0f) * (19.0f - 44.0f * x + 24.0f * x2 + 16.0f * x * x2 - 16.0f * x4);
    w[2] = (1.0f / 192.0f) * (115.0f - 120.0f * x2 + 48.0f * x4);
    w[3] = (1.0f / 96.0f) * (19.0f + 44.0f * x + 24.0f * x2 - 16.0f * x * x2 - 16.0f * x4);
    w[4] = (1.0f / 384.0f) * (1.0f + 8.0f * x + 24.0f * x2 + 32.0f * x * x2 + 16.0f * x4);
}

__device__ __forceinline__ int wrapi(int p, int n) {
    p %= n;
    return p < 0 ? p + n : p;
}

struct P3MGeom {
    int3 sz;
    float3 lo, h, invh;
    float qunit;
};

__device__ __forceinline__ void stencil(const P3MGeom &g, float4 x, int3 &ng, float3 &d) {
    const float px = x.x - g.lo.x, py = x.y - g.lo.y, pz = x.z - g.lo.z;
    ng.x = (int)floorf((px + 0.5f * g.h.x) / g.h.x);
    ng.y = (int)floorf((py + 0.5f * g.h.y) / g.h.y);
    ng.z = (int)floorf((pz + 0.5f * g.h.z) / g.h.z);
    d.x = px / g.h.x - (float)ng.x;
    d.y = py / g.h.y - (float)ng.y;
    d.z = pz / g.h.z - (float)ng.z;
}

// Arguments of the P3M kernels for one system: a0 (single system) or
// tab[blockIdx.y] (batched replicas; a0 then only sizes the grid).
struct P3MArgs {
    int n;
    const float4 *xs;
    const float *qs;
    float4 *fs;
    P3MGeom g;
    float *rho;
    const float2 *rho_k;
    float2 *e_k;
    const float *e_r;
    const float *green;
    float3 tpl;  // 2 pi / L
    size_t nk, ngrid;
    float niv;   // -1 / V
    // molecule form (all-rigid water): the charged sites of molecule m are
    // H1, H2, M of mol_idx[m] (four-site, uncharged O) or O, H1, H2
    const int4 *mol_idx;
    int nmol, four_site;
    int slots;  // 1: the molecule form's layout, molecule slot m at sites 4m .. 4m+3 (no map read)
    const float4 *e4;  // the own FFT's interleaved field (batched gather), or null
};
#define MDX_P3M_ARGS const P3MArgs A = tab ? tab[blockIdx.y] : a0

// map_charge_to_grid_order_5_cu (FixChargeEwald.cu:174-217) with five lanes
// per atom: lane t adds the 25 points of stencil plane a = t.  The six atoms
// of a warp are taken W = n/6 apart (atom g W + warp) so that the float
// atomics of one warp instruction land in distant parts of the mesh instead
// of piling onto the same points (neighbouring atoms are adjacent in the
// cell-sorted order)
__device__ __forceinline__ float pick5(const float w[5], int t) {
    return t == 0 ? w[0] : t == 1 ? w[1] : t == 2 ? w[2] : t == 3 ? w[3] : w[4];
}

// stencil plane a = t of atom i's charge (25 points, as two 16-byte vector
// atomics per z row: the five z points lie in two aligned groups of four,
// the mesh side being a multiple of 4)
__device__ __forceinline__ void spread_plane(const P3MArgs &A, int i, int t) {
    const float q = A.qs[i];
    if (q == 0.f) return;
    const P3MGeom &g = A.g;
    const float qi = g.qunit * q;
    int3 ng;
    float3 d;
    stencil(g, A.xs[i], ng, d);
    float wx[5], wy[5], wz[5];
    w5(d.x, wx);
    w5(d.y, wy);
    w5(d.z, wz);
    int pz[5];
#pragma unroll
    for (int c = 0; c < 5; c++) pz[c] = wrapi(ng.z + c - 2, g.sz.z);
    const int px = wrapi(ng.x + t - 2, g.sz.x);
    const float cyz = qi * pick5(wx, t);
    const int z0 = pz[0], g0 = z0 & ~3, sh = z0 - g0;
    const int g1 = (g0 + 4) % g.sz.z;
#pragma unroll
    for (int b = 0; b < 5; b++) {
        const int py = wrapi(ng.y + b - 2, g.sz.y);
        const float cz = cyz * wy[b];
        float w[5];
#pragma unroll
        for (int c = 0; c < 5; c++) w[c] = cz * wz[c];
        float4 v1, v2;
        switch (sh) {
            case 0: v1 = make_float4(w[0], w[1], w[2], w[3]); v2 = make_float4(w[4], 0.f, 0.f, 0.f); break;
            case 1: v1 = make_float4(0.f, w[0], w[1], w[2]); v2 = make_float4(w[3], w[4], 0.f, 0.f); break;
            case 2: v1 = make_float4(0.f, 0.f, w[0], w[1]); v2 = make_float4(w[2], w[3], w[4], 0.f); break;
            default: v1 = make_float4(0.f, 0.f, 0.f, w[0]); v2 = make_float4(w[1], w[2], w[3], w[4]); break;
        }
        float *row = A.rho + ((size_t)px * g.sz.y + py) * g.sz.z;
        atomicAdd(reinterpret_cast<float4 *>(row + g0), v1);
        atomicAdd(reinterpret_cast<float4 *>(row + g1), v2);
    }
}

__global__ void k_spread5(const P3MArgs a0, const P3MArgs *__restrict__ tab) {
    pdl_wait();
    MDX_P3M_ARGS;
    const int lane = threadIdx.x & 31;
    const int t = lane % 5;
    const int W = (A.n + 5) / 6;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int i = (lane / 5) * W + w;
    if (lane >= 30 || w >= W || i >= A.n) return;
    spread_plane(A, i, t);
}

__device__ __forceinline__ int mol_site(int4 ix, int k, int four_site) {
    return four_site ? (k == 0 ? ix.y : (k == 1 ? ix.z : ix.w)) : (k == 0 ? ix.x : (k == 1 ? ix.y : ix.z));
}
__device__ __forceinline__ int4 mol_atoms(const P3MArgs &A, int m) {
    return A.slots ? make_int4(4 * m, 4 * m + 1, 4 * m + 2, 4 * m + 3) : A.mol_idx[m];
}

// the molecule form: lanes 15 j .. 15 j + 14 of a warp take the three
// charged sites (five planes each) of one molecule, two molecules per warp,
// the two W = nmol/2 apart; no lane is spent on an uncharged oxygen
__global__ void k_spread_mol(const P3MArgs a0, const P3MArgs *__restrict__ tab) {
    pdl_wait();
    MDX_P3M_ARGS;
    const int lane = threadIdx.x & 31;
    const int W = (A.nmol + 1) / 2;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int m = (lane / 15) * W + w;
    if (lane >= 30 || w >= W || m >= A.nmol) return;
    spread_plane(A, mol_site(mol_atoms(A, m), (lane % 15) / 5, A.four_site), lane % 5);
}

// E_d(k) = i k_d G rho on the half spectrum (z halved), batched output
__global__ void k_efield(const P3MArgs a0, const P3MArgs *__restrict__ tab) {
    MDX_P3M_ARGS;
    const size_t nk = A.nk;
    size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nk) return;
    const int3 sz = A.g.sz;
    const float3 twopi_over_L = A.tpl;
    const float2 *__restrict__ rho_k = A.rho_k;
    const float *__restrict__ green = A.green;
    float2 *__restrict__ ek = A.e_k;
    const int nzh = sz.z / 2 + 1;
    const int iz = (int)(id % nzh);
    const int iy = (int)((id / nzh) % sz.y);
    const int ix = (int)(id / ((size_t)nzh * sz.y));
    const float kx = twopi_over_L.x * (float)(ix > sz.x / 2 ? ix - sz.x : ix);
    const float ky = twopi_over_L.y * (float)(iy > sz.y / 2 ? iy - sz.y : iy);
    const float kz = twopi_over_L.z * (float)iz;
    const float G = green[id];
    const float2 q = rho_k[id];
    // i k G (q.x + i q.y) = (-k G q.y) + i (k G q.x); Nyquist planes dropped per component
    const float gx = (2 * ix == sz.x) ? 0.f : kx * G;
    const float gy = (2 * iy == sz.y) ? 0.f : ky * G;
    const float gz = (2 * iz == sz.z) ? 0.f : kz * G;
    ek[id] = make_float2(-gx * q.y, gx * q.x);
    ek[nk + id] = make_float2(-gy * q.y, gy * q.x);
    ek[2 * nk + id] = make_float2(-gz * q.y, gz * q.x);
}

template <bool ACC>
__global__ void k_gather(const P3MArgs a0, const P3MArgs *__restrict__ tab) {
    MDX_P3M_ARGS;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    const float4 *__restrict__ xs = A.xs;
    const float *__restrict__ qs = A.qs;
    const P3MGeom &g = A.g;
    const float *__restrict__ er = A.e_r;
    const size_t ngrid = A.ngrid;
    const float neg_inv_vol = A.niv;
    float4 *__restrict__ fs = A.fs;
    const float q = qs[i];
    if (q == 0.f) {
        if (!ACC) {
            float4 f = fs[i];
            fs[i] = make_float4(0.f, 0.f, 0.f, f.w);
        }
        return;
    }
    int3 ng;
    float3 d;
    stencil(g, xs[i], ng, d);
    float wx[5], wy[5], wz[5];
    w5(d.x, wx);
    w5(d.y, wy);
    w5(d.z, wz);
    int pz[5];
#pragma unroll
    for (int c = 0; c < 5; c++) pz[c] = wrapi(ng.z + c - 2, g.sz.z);
    float ex = 0.f, ey = 0.f, ez = 0.f;
#pragma unroll
    for (int a = 0; a < 5; a++) {
        const int px = wrapi(ng.x + a - 2, g.sz.x);
#pragma unroll
        for (int b = 0; b < 5; b++) {
            const int py = wrapi(ng.y + b - 2, g.sz.y);
            const size_t row = ((size_t)px * g.sz.y + py) * g.sz.z;
            const float wab = wx[a] * wy[b];
#pragma unroll
            for (int c = 0; c < 5; c++) {
                const float w = wab * wz[c];
                const size_t o = row + pz[c];
                ex += w * __ldg(er + o);
                ey += w * __ldg(er + ngrid + o);
                ez += w * __ldg(er + 2 * ngrid + o);
            }
        }
    }
    const float s = g.qunit * q * neg_inv_vol;
    float4 f = fs[i];
    if (ACC) {
        f.x += s * ex;
        f.y += s * ey;
        f.z += s * ez;
    } else {
        f.x = s * ex;
        f.y = s * ey;
        f.z = s * ez;
    }
    fs[i] = f;
}

// sum_k G |rho_k|^2 over the full spectrum from the half spectrum (FP64)
__global__ void k_recip_energy(int3 sz, const float2 *__restrict__ rho_k, const float *__restrict__ green, size_t nk,
                               double *out) {
    double acc = 0.0;
    const int nzh = sz.z / 2 + 1;
    for (size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x; id < nk; id += (size_t)gridDim.x * blockDim.x) {
        const int iz = (int)(id % nzh);
        const double w = (iz == 0 || 2 * iz == sz.z) ? 1.0 : 2.0;
        const float2 q = rho_k[id];
        acc += w * (double)green[id] * ((double)q.x * q.x + (double)q.y * q.y);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, acc);
}

// virials_cu (FixChargeEwald.cu:731-812) on the half spectrum: the 6-vector
// sum_k w G |rho_k|^2 (delta_ab - 2 (1/k^2 + 1/(4 alpha^2)) k_a k_b), k != 0,
// w = 2 for the kz planes that stand for their conjugates; FP64 sums
__global__ void k_recip_virial(int3 sz, const float2 *__restrict__ rho_k, const float *__restrict__ green, size_t nk,
                               double3 tpl, double alpha, double *out) {
    double acc[6] = {0, 0, 0, 0, 0, 0};
    const int nzh = sz.z / 2 + 1;
    const double f4a = 0.25 / (alpha * alpha);
    for (size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x; id < nk; id += (size_t)gridDim.x * blockDim.x) {
        const int iz = (int)(id % nzh);
        const int iy = (int)((id / nzh) % sz.y);
        const int ix = (int)(id / ((size_t)nzh * sz.y));
        const double kx = tpl.x * (ix > sz.x / 2 ? ix - sz.x : ix);
        const double ky = tpl.y * (iy > sz.y / 2 ? iy - sz.y : iy);
        const double kz = tpl.z * iz;
        const double k2 = kx * kx + ky * ky + kz * kz;
        if (k2 == 0.0) continue;
        const double w = (iz == 0 || 2 * iz == sz.z) ? 1.0 : 2.0;
        const float2 q = rho_k[id];
        const double E = w * (double)green[id] * ((double)q.x * q.x + (double)q.y * q.y);
        const double d = -2.0 * (1.0 / k2 + f4a);
        acc[0] += (1.0 + d * kx * kx) * E;
        acc[1] += (1.0 + d * ky * ky) * E;
        acc[2] += (1.0 + d * kz * kz) * E;
        acc[3] += d * kx * ky * E;
        acc[4] += d * kx * kz * E;
        acc[5] += d * ky * kz * E;
    }
#pragma unroll
    for (int c = 0; c < 6; c++) {
        double v = acc[c];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) atomicAdd(out + c, v);
    }
}

// mapVirialToSingleAtom (FixChargeEwald.cu:815-818): the field virial, 0.5/V
// of the sum, goes onto the first atom's per-atom virial
__global__ void k_add_field_virial(float *__restrict__ vir, const double *__restrict__ sum6, double scale) {
    const int c = threadIdx.x;
    if (c < 6) vir[c] += (float)(scale * sum6[c]);
}

__host__ __device__ double sinc(double x) {
    if (x < 0.1 && x > -0.1) {
        double x2 = x * x;
        return 1.0 - x2 * 0.16666666667 + x2 * x2 * 0.008333333333333333 - x2 * x2 * x2 * 0.00019841269841269841;
    }
    return std::sin(x) / x;
}

const double kAmp[5][5] = {
    {2.0 / 3.0, 0, 0, 0, 0},
    {1.0 / 50.0, 5.0 / 294.0, 0, 0, 0},
    {1.0 / 588.0, 7.0 / 1440.0, 21.0 / 3872.0, 0, 0},
    {1.0 / 4320.0, 3.0 / 1936.0, 7601.0 / 2271360.0, 143.0 / 28800.0, 0},
    {1.0 / 23232.0, 7601.0 / 12628160.0, 143.0 / 69120.0, 517231.0 / 106536960.0, 106640677.0 / 11737571328.0},
};

P3MGeom geom(State &s, FixChargeEwald &f) {
    P3MGeom g;
    g.sz = f.sz;
    g.lo = s.box.lo;
    g.h = make_float3(s.box.L.x / (float)f.sz.x, s.box.L.y / (float)f.sz.y, s.box.L.z / (float)f.sz.z);
    g.invh = make_float3(1.f / g.h.x, 1.f / g.h.y, 1.f / g.h.z);
    g.qunit = (float)std::sqrt(s.units.qqr_to_eng);
    return g;
}

P3MArgs p3m_args(State &s, FixChargeEwald &f) {
    P3MArgs A{};
    A.n = s.gpd.n;
    A.xs = s.gpd.xs.p;
    A.qs = s.gpd.qs.p;
    A.fs = s.gpd.fs.p;
    A.g = geom(s, f);
    A.rho = f.rho.p;
    A.rho_k = f.rho_k.p;
    A.e_k = f.e_k.p;
    A.e_r = f.e_r.p;
    A.green = f.green.p;
    A.tpl = make_float3((float)(6.28318530717958647693 / s.box.Ld.x), (float)(6.28318530717958647693 / s.box.Ld.y),
                        (float)(6.28318530717958647693 / s.box.Ld.z));
    A.nk = (size_t)f.sz.x * f.sz.y * (f.sz.z / 2 + 1);
    A.ngrid = (size_t)f.sz.x * f.sz.y * f.sz.z;
    A.niv = (float)(-1.0 / (s.box.Ld.x * s.box.Ld.y * s.box.Ld.z));
    A.slots = 0;
    A.e4 = f.own_fft ? f.e4.p : nullptr;
    return A;
}

// ---- P3M reciprocal solve on our own FFT (cubic 32^3, 64^3, 128^3 meshes) --
// A line of N points is transformed by TL = 8 lanes of a warp (four lines per
// warp), each holding P = N/8 points: a P-point DFT in registers over the
// points TL n1 + l of lane l, twiddles W_N^(l k1), one exchange of the line
// among its lanes through shared memory, then P/TL DFTs of TL points over the
// lanes' index.  Lane l ends with X[(l + TL m) + P k2] in v[m TL + k2]; the
// inverse runs the same steps backwards, from that layout to the points
// TL n1 + l, so neither direction permutes a line beyond its one exchange.
// Unnormalised, as cuFFT.  (One line per warp with five radix-2 shuffle
// stages, the layout before, spent 20 shuffles and as many selects per line
// and lane, and read and wrote one 8-byte word per 32-byte sector in the x
// pass; figures at own_solve.)
// Three kernels replace R2C + E(k) + batched C2R:
//   k_fft_zy   per x plane: real FFTs along z, two rows packed into one
//              complex transform (half spectrum kept), then along y
//   k_fft_xe   per (kz, 32/TL adjacent ky): FFT along x, E_d(k) = i k_d G rho
//              (Nyquist planes dropped per component, as k_efield), 3 inverse
//              FFTs along x; whole 32-byte sectors on both sides
//   k_ifft_yz  per x plane, (Ex, Ey) or Ez: inverse along y, then along z
//              with (Ex, Ey) of a row, or Ez of two rows, packed into one
//              complex transform; E interleaved as float4 (Ex, Ey, Ez, unset)
// so the gather reads one 16-byte value per stencil point.
struct FFTArgs {
    int n;                   // points per side (32, 64 or 128)
    const float *rho;        // [n][n][n]
    float2 *mid1;            // [n][n/2+1][n] (x, kz, ky): after the z and y passes
    float2 *mid2;            // [3][n][n/2+1][n] (d, x, kz, ky): E_d after the inverse x pass
    float4 *e4;              // [n][n][n]
    const float *green;      // [n][n/2+1][n] (kx, kz, ky)
    const float2 *tw;        // W_n^k, forward sign
    float3 tpl;              // 2 pi / L
};

__device__ __forceinline__ float2 operator+(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 operator-(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// times -i (forward) or i (inverse)
template <bool INV>
__device__ __forceinline__ float2 rot90(float2 a) {
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
// times w (forward sign given) or its conjugate
template <bool INV>
__device__ __forceinline__ float2 twid(float2 a, float2 w) {
    return INV ? make_float2(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y) : cmul(a, w);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2 &a, float2 &b, float2 &c, float2 &d) {
    const float2 s0 = a + c, s1 = a - c, s2 = b + d, s3 = rot90<INV>(b - d);
    a = s0 + s2;
    b = s1 + s3;
    c = s0 - s2;
    d = s1 - s3;
}

// DFT of the n values v[0], ..., v[n-1] in place (n = 4, 8, 16)
template <int n, bool INV>
__device__ __forceinline__ void dft(float2 *v) {
    constexpr float kR = 0.70710678118654752f;   // cos(pi/4)
    constexpr float kC = 0.92387953251128674f;   // cos(pi/8)
    constexpr float kS = 0.38268343236508977f;   // sin(pi/8)
    if constexpr (n == 4) {
        dft4<INV>(v[0], v[1], v[2], v[3]);
    } else if constexpr (n == 8) {
        float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        dft4<INV>(e[0], e[1], e[2], e[3]);
        dft4<INV>(o[0], o[1], o[2], o[3]);
        o[1] = twid<INV>(o[1], make_float2(kR, -kR));
        o[2] = rot90<INV>(o[2]);
        o[3] = twid<INV>(o[3], make_float2(-kR, -kR));
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = e[k] + o[k];
            v[k + 4] = e[k] - o[k];
        }
    } else {
        static_assert(n == 16, "4, 8 or 16 points");
        const float2 w1 = make_float2(kC, -kS), w2 = make_float2(kR, -kR), w3 = make_float2(kS, -kC);
        float2 y[4][4];  // y[b][k1]: DFT over a of v[4 a + b]
#pragma unroll
        for (int b = 0; b < 4; b++) {
#pragma unroll
            for (int a = 0; a < 4; a++) y[b][a] = v[4 * a + b];
            dft4<INV>(y[b][0], y[b][1], y[b][2], y[b][3]);
        }
        // times W_16^(b k1)
        y[1][1] = twid<INV>(y[1][1], w1);
        y[1][2] = twid<INV>(y[1][2], w2);
        y[1][3] = twid<INV>(y[1][3], w3);
        y[2][1] = twid<INV>(y[2][1], w2);
        y[2][2] = rot90<INV>(y[2][2]);
        y[2][3] = twid<INV>(y[2][3], make_float2(-kR, -kR));
        y[3][1] = twid<INV>(y[3][1], w3);
        y[3][2] = twid<INV>(y[3][2], make_float2(-kR, -kR));
        y[3][3] = twid<INV>(y[3][3], make_float2(-kC, kS));
#pragma unroll
        for (int k1 = 0; k1 < 4; k1++) {
            dft4<INV>(y[0][k1], y[1][k1], y[2][k1], y[3][k1]);
#pragma unroll
            for (int k2 = 0; k2 < 4; k2++) v[k1 + 4 * k2] = y[k2][k1];
        }
    }
}

template <int N>
struct Line {
    static constexpr int TL = 8;         // lanes per line
    static constexpr int P = N / TL;     // points per lane
    static constexpr int LPW = 32 / TL;  // lines per warp
    static constexpr int NH = N / 2 + 1;
    // n = 32: fewer points per lane than lanes, so two lanes share each
    // second-stage transform (its even and odd outputs)
    static constexpr bool PAIR = P < TL;
    static constexpr int M2 = PAIR ? 1 : P / TL;  // second-stage DFTs per lane
    // row pitch of a plane in shared memory: 2 modulo 16 complex words, so
    // that a column's eight lanes and two adjacent columns hit all banks, and
    // two rows hold a line of N
    static constexpr int PITCH = NH + 1;
    // where value (k1, n2) of a line sits during the exchange: rows of TL
    // values, rotated so that both the writes (n2 across lanes) and the reads
    // (k1 across lanes) spread over the banks
    static __device__ __forceinline__ int slot(int k1, int n2) { return k1 * TL + ((n2 + k1) & (TL - 1)); }
    // the frequency in v[j] of lane l
    static __device__ __forceinline__ int freq(int j, int l) {
        return PAIR ? (l >> 1) + P * (2 * j + (l & 1)) : l + TL * (j / TL) + P * (j % TL);
    }
};

// times W_8^n (forward sign) or its conjugate, n = 0 .. 3 known at compile time
template <bool INV>
__device__ __forceinline__ float2 w8(float2 a, int n) {
    constexpr float kR = 0.70710678118654752f;
    return n == 0 ? a : (n == 1 ? twid<INV>(a, make_float2(kR, -kR)) : (n == 2 ? rot90<INV>(a)
                                                                               : twid<INV>(a, make_float2(-kR, -kR))));
}

// buf(pos): the line's exchange buffer, N words that its lanes own; the
// warp's lanes call together (idle lines carry zeros and touch no buffer)
template <int N, class Buf>
__device__ __forceinline__ void fft_line(float2 (&v)[Line<N>::P], int l, bool active, const float2 *__restrict__ tw,
                                         Buf buf) {
    using F = Line<N>;
    dft<F::P, false>(v);
#pragma unroll
    for (int k1 = 1; k1 < F::P; k1++) v[k1] = cmul(v[k1], __ldg(tw + l * k1));
    if (active)
#pragma unroll
        for (int k1 = 0; k1 < F::P; k1++) buf(F::slot(k1, l)) = v[k1];
    __syncwarp();
    if constexpr (F::PAIR) {
        // X[k1 + P (2 j + h)] = DFT_P over n of W_8^(n h) (z[n] +- z[n + P])
        if (active)
#pragma unroll
            for (int n = 0; n < F::P; n++) {
                const float2 a = buf(F::slot(l >> 1, n)), b = buf(F::slot(l >> 1, n + F::P));
                v[n] = l & 1 ? w8<false>(a - b, n) : a + b;
            }
        __syncwarp();
        dft<F::P, false>(v);
    } else {
        if (active)
#pragma unroll
            for (int m = 0; m < F::M2; m++)
#pragma unroll
                for (int n2 = 0; n2 < F::TL; n2++) v[m * F::TL + n2] = buf(F::slot(l + F::TL * m, n2));
        __syncwarp();
#pragma unroll
        for (int m = 0; m < F::M2; m++) dft<F::TL, false>(v + m * F::TL);
    }
}

template <int N, class Buf>
__device__ __forceinline__ void ifft_line(float2 (&v)[Line<N>::P], int l, bool active, const float2 *__restrict__ tw,
                                          Buf buf) {
    using F = Line<N>;
    if constexpr (F::PAIR) {
        // the even and the odd frequencies' transforms c_0, c_1 by two lanes;
        // z[n2] = c_0[n2 mod P] + W_8^-n2 c_1[n2 mod P]
        dft<F::P, true>(v);
        if (active)
#pragma unroll
            for (int n = 0; n < F::P; n++) buf(F::slot(l >> 1, (l & 1) * F::P + n)) = v[n];
        __syncwarp();
        if (active) {
            const float2 w = __ldg(tw + F::P * l);
#pragma unroll
            for (int k1 = 0; k1 < F::P; k1++) {
                const float2 c0 = buf(F::slot(k1, l & (F::P - 1))), c1 = buf(F::slot(k1, F::P + (l & (F::P - 1))));
                v[k1] = twid<true>(c0 + twid<true>(c1, w), __ldg(tw + l * k1));
            }
        }
        __syncwarp();
    } else {
#pragma unroll
        for (int m = 0; m < F::M2; m++) {
            dft<F::TL, true>(v + m * F::TL);
#pragma unroll
            for (int n2 = 1; n2 < F::TL; n2++)
                v[m * F::TL + n2] = twid<true>(v[m * F::TL + n2], __ldg(tw + (l + F::TL * m) * n2));
        }
        if (active)
#pragma unroll
            for (int m = 0; m < F::M2; m++)
#pragma unroll
                for (int n2 = 0; n2 < F::TL; n2++) buf(F::slot(l + F::TL * m, n2)) = v[m * F::TL + n2];
        __syncwarp();
        if (active)
#pragma unroll
            for (int k1 = 0; k1 < F::P; k1++) v[k1] = buf(F::slot(k1, l));
        __syncwarp();
    }
    dft<F::P, true>(v);
}

// threads per block of the plane kernels: forward, one line per group for the
// n/2 row pairs and (a warp more) the n/2+1 columns; inverse, the 2 (n/2+1)
// columns of part 0 in one round (two at n = 128)
template <int N>
constexpr int kZyThreads = N / 2 * Line<N>::TL + 32;
template <int N>
constexpr int kYzThreads = N == 32 ? 288 : 544;

template <int N>
__global__ void __launch_bounds__(kZyThreads<N>) k_fft_zy(const FFTArgs a0, const FFTArgs *__restrict__ tab) {
    extern __shared__ float2 plane[];  // [n][PITCH]
    using F = Line<N>;
    constexpr int TL = F::TL, P = F::P, NH = F::NH, PITCH = F::PITCH;
    pdl_wait();
    const FFTArgs A = tab ? tab[blockIdx.y] : a0;  // batched replicas: blockIdx.y
    const int x = blockIdx.x;
    const int l = threadIdx.x % TL, line = threadIdx.x / TL;
    {
        // rows 2 line and 2 line + 1 as one complex line (plain loads: the
        // spread may still be writing the mesh when this grid starts, and the
        // read-only path promises data that no one writes while it runs)
        const bool active = line < N / 2;
        float2 v[P];
        const float *r0 = A.rho + ((size_t)x * N + 2 * (active ? line : 0)) * N + l;
#pragma unroll
        for (int n1 = 0; n1 < P; n1++) v[n1] = make_float2(r0[TL * n1], r0[N + TL * n1]);
        float2 *const row = plane + 2 * (active ? line : 0) * PITCH;
        auto buf = [&](int pos) -> float2 & { return row[pos]; };
        fft_line<N>(v, l, active, A.tw, buf);
        if (active)
#pragma unroll
            for (int j = 0; j < P; j++) row[F::freq(j, l)] = v[j];
        __syncwarp();
        // Z = FFT(a + i b): A = (Z[k] + conj Z[-k]) / 2, B = (Z[k] - conj Z[-k]) / 2i
        constexpr int H = P / 2;  // k = l, l + TL, ..., below n/2, and n/2 itself by lane 0
        float2 a[H + 1], b[H + 1];
#pragma unroll
        for (int i = 0; i <= H; i++) {
            const int k = l + TL * i;
            const float2 p = active && k < NH ? row[k] : make_float2(0.f, 0.f);
            const float2 q = active && k < NH ? row[(N - k) & (N - 1)] : make_float2(0.f, 0.f);
            a[i] = make_float2(0.5f * (p.x + q.x), 0.5f * (p.y - q.y));
            b[i] = make_float2(0.5f * (p.y + q.y), 0.5f * (q.x - p.x));
        }
        __syncwarp();
        if (active)
#pragma unroll
            for (int i = 0; i <= H; i++) {
                const int k = l + TL * i;
                if (k < NH) {
                    row[k] = a[i];
                    row[PITCH + k] = b[i];
                }
            }
    }
    __syncthreads();
    {
        const bool active = line < NH;
        const int kz = active ? line : 0;
        float2 v[P];
#pragma unroll
        for (int n1 = 0; n1 < P; n1++)
            v[n1] = active ? plane[(TL * n1 + l) * PITCH + kz] : make_float2(0.f, 0.f);
        __syncwarp();
        auto buf = [&](int pos) -> float2 & { return plane[pos * PITCH + kz]; };
        fft_line<N>(v, l, active, A.tw, buf);
        float2 *out = A.mid1 + ((size_t)x * NH + kz) * N;
        if (active)
#pragma unroll
            for (int j = 0; j < P; j++) out[F::freq(j, l)] = v[j];
    }
}

constexpr int kXeWarps = 2;

template <int N>
__global__ void __launch_bounds__(kXeWarps * 32) k_fft_xe(const FFTArgs a0, const FFTArgs *__restrict__ tab) {
    using F = Line<N>;
    constexpr int TL = F::TL, P = F::P, NH = F::NH, LPW = F::LPW;
    __shared__ float2 sh[kXeWarps][N * LPW];
    pdl_wait();
    const FFTArgs A = tab ? tab[blockIdx.y] : a0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int task = blockIdx.x * kXeWarps + w;
    if (task >= NH * (N / LPW)) return;  // warp-uniform; no block barrier below
    const int sub = lane % LPW, l = lane / LPW;
    const int kz = task / (N / LPW), ky = task % (N / LPW) * LPW + sub;
    float2 *const line = sh[w];
    auto buf = [&](int pos) -> float2 & { return line[pos * LPW + sub]; };
    const size_t at = (size_t)kz * N + ky;
    constexpr size_t stride = (size_t)NH * N;
    float2 q[P];
#pragma unroll
    for (int n1 = 0; n1 < P; n1++) q[n1] = A.mid1[(TL * n1 + l) * stride + at];
    float G[P];
#pragma unroll
    for (int j = 0; j < P; j++) G[j] = __ldg(A.green + F::freq(j, l) * stride + at);
    fft_line<N>(q, l, true, A.tw, buf);
    const float kyv = 2 * ky == N ? 0.f : A.tpl.y * (float)(ky > N / 2 ? ky - N : ky);
    const float kzv = 2 * kz == N ? 0.f : A.tpl.z * (float)kz;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        float2 u[P];
#pragma unroll
        for (int j = 0; j < P; j++) {
            const int kx = F::freq(j, l);
            const float kxv = 2 * kx == N ? 0.f : A.tpl.x * (float)(kx > N / 2 ? kx - N : kx);
            const float g = (d == 0 ? kxv : (d == 1 ? kyv : kzv)) * G[j];
            u[j] = make_float2(-g * q[j].y, g * q[j].x);
        }
        ifft_line<N>(u, l, true, A.tw, buf);
        float2 *out = A.mid2 + (size_t)d * N * stride + at;
#pragma unroll
        for (int n1 = 0; n1 < P; n1++) out[(TL * n1 + l) * stride] = u[n1];
    }
}

// one block per (x plane, part): part 0 the components x and y, part 1 z.
// Along z, a line of a + i b from the half spectra of two real rows a and b,
// extended by X[n - k] = conj X[k]: (Ex, Ey) of a row, or Ez of two rows
template <int N, int D>
__device__ __forceinline__ void ifft_yz_part(const FFTArgs &A, float2 *plane) {
    using F = Line<N>;
    constexpr int TL = F::TL, P = F::P, NH = F::NH, PITCH = F::PITCH;
    constexpr int kLines = kYzThreads<N> / TL;
    constexpr int kRoundsY = (D * NH + kLines - 1) / kLines;
    constexpr int kLinesZ = D == 2 ? N : N / 2, kRoundsZ = (kLinesZ + kLines - 1) / kLines;
    const int x = blockIdx.x;
    const int l = threadIdx.x % TL, line = threadIdx.x / TL;
    constexpr size_t stride = (size_t)NH * N;
#pragma unroll 1
    for (int r = 0; r < kRoundsY; r++) {
        const int t = line + r * kLines;
        const bool active = t < D * NH;
        const int d = active ? t / NH : 0, kz = active ? t % NH : 0;
        float2 v[P];
        const float2 *src = A.mid2 + ((size_t)(D == 2 ? d : 2) * N + x) * stride + (size_t)kz * N;
#pragma unroll
        for (int j = 0; j < P; j++) v[j] = src[F::freq(j, l)];
        float2 *const col = plane + (size_t)d * N * PITCH + kz;
        auto buf = [&](int pos) -> float2 & { return col[pos * PITCH]; };
        ifft_line<N>(v, l, active, A.tw, buf);
        if (active)
#pragma unroll
            for (int n1 = 0; n1 < P; n1++) col[(TL * n1 + l) * PITCH] = v[n1];
    }
    __syncthreads();
#pragma unroll 1
    for (int r = 0; r < kRoundsZ; r++) {
        const int t = line + r * kLines;
        const bool active = t < kLinesZ;
        // D = 2: row t of both planes; D = 1: rows 2t and 2t + 1
        float2 *const ra = plane + (size_t)(active ? (D == 2 ? t : 2 * t) : 0) * PITCH;
        float2 *const rb = ra + (D == 2 ? (size_t)N * PITCH : (size_t)PITCH);
        float2 v[P];
#pragma unroll
        for (int j = 0; j < P; j++) {
            const int k = F::freq(j, l), kk = k <= N / 2 ? k : N - k;
            float2 a = active ? ra[kk] : make_float2(0.f, 0.f), b = active ? rb[kk] : make_float2(0.f, 0.f);
            if (k == 0 || k == N / 2) a.y = b.y = 0.f;
            if (k > N / 2) {
                a.y = -a.y;
                b.y = -b.y;
            }
            v[j] = make_float2(a.x - b.y, a.y + b.x);
        }
        __syncwarp();
        // the two rows' words are the exchange buffer: one half line in each
        auto buf = [&](int pos) -> float2 & { return pos < N / 2 ? ra[pos] : rb[pos - N / 2]; };
        ifft_line<N>(v, l, active, A.tw, buf);
        if (!active) continue;  // no warp barrier below
        float *out = reinterpret_cast<float *>(A.e4 + ((size_t)x * N + (D == 2 ? t : 2 * t)) * N + l);
        if (D == 2) {
#pragma unroll
            for (int n1 = 0; n1 < P; n1++) *reinterpret_cast<float2 *>(out + 4 * TL * n1) = v[n1];
        } else {
#pragma unroll
            for (int n1 = 0; n1 < P; n1++) {
                out[4 * TL * n1 + 2] = v[n1].x;
                out[4 * (N + TL * n1) + 2] = v[n1].y;
            }
        }
    }
}

template <int N>
__global__ void __launch_bounds__(kYzThreads<N>) k_ifft_yz(const FFTArgs a0, const FFTArgs *__restrict__ tab) {
    extern __shared__ float2 plane[];  // [2][n][PITCH]
    pdl_wait();
    const FFTArgs A = tab ? tab[blockIdx.z] : a0;  // batched replicas: blockIdx.z
    if (blockIdx.y == 0) ifft_yz_part<N, 2>(A, plane);
    else ifft_yz_part<N, 1>(A, plane);
}

// the three kernels for one system (a0) or the nrep systems of tab
template <int N, class Launch>
void launch_solve(Launch launch, unsigned nrep) {
    using F = Line<N>;
    constexpr size_t row = (size_t)N * F::PITCH * sizeof(float2);
    launch(k_fft_zy<N>, dim3(N, nrep), dim3(kZyThreads<N>), row);
    launch(k_fft_xe<N>, dim3((F::NH * (N / F::LPW) + kXeWarps - 1) / kXeWarps, nrep), dim3(kXeWarps * 32), (size_t)0);
    launch(k_ifft_yz<N>, dim3(N, 2, nrep), dim3(kYzThreads<N>), 2 * row);
}

// Gather on the interleaved field: a warp takes three charges -- the charged
// sites of one molecule (MOL; no lane is spent on an uncharged oxygen) or
// three consecutive atoms.  Lane 3 s + d works out charge s's stencil along
// dimension d once, into shared memory; then a charge's 125 points go over
// the lanes in mesh order (four 16-byte loads a lane, the twelve of the three
// charges in flight), so that a load instruction reads runs of 80 bytes and
// touches about 8 lines; the nine sums are butterflied.  What bounds it is the
// L2's bandwidth: 75 rows of 80 bytes per molecule, 34 MB at 4,096 molecules.
// A lane per stencil plane, the layout before, touched one 32-byte sector
// per point (49 MB): gather stage of 8,000 atoms on 32^3 12.8 -> 10.8 us, of
// 32,768 molecules on 128^3 (planar fields then, one thread per site) with the
// chain, see own_solve.  Neighbouring molecules go to one block for its L1.
// MOL: stored into a per-step buffer, the uncharged oxygen of a four-site
// molecule as zero; otherwise stored into (ACC: added to) the forces, whose .w
// is kept.  Batched replicas (blockIdx.y): each its own field.
constexpr int kMeshWarps = 4;  // warps per block

struct Stencil {
    float wx[3][5], wy[3][5], wz[3][5];  // weights
    int ox[3][5], oy[3][5], pz[3][5];    // offset of plane a, of row b within it, index of point c
    float q[3];
};

template <bool MOL>
__device__ __forceinline__ int unit_atom(const P3MArgs &A, int u, int s) {
    if (MOL) return mol_site(mol_atoms(A, u), s, A.four_site);
    return 3 * u + s < A.n ? 3 * u + s : -1;
}
template <bool MOL>
__host__ __device__ __forceinline__ int mesh_units(int n, int nmol) {
    return MOL ? nmol : (n + 2) / 3;
}
template <bool MOL>
unsigned mesh_blocks(int n, int nmol) {
    return (unsigned)((mesh_units<MOL>(n, nmol) + kMeshWarps - 1) / kMeshWarps);
}

template <bool MOL, bool ACC>
__global__ void __launch_bounds__(kMeshWarps * 32) k_gather4(const P3MArgs a0, const P3MArgs *__restrict__ tab) {
    __shared__ Stencil sh[kMeshWarps];
    pdl_wait();
    MDX_P3M_ARGS;
    const int u = blockIdx.x * kMeshWarps + (threadIdx.x >> 5);
    if (u >= mesh_units<MOL>(A.n, A.nmol)) return;  // warp-uniform
    const int lane = threadIdx.x & 31;
    Stencil &S = sh[threadIdx.x >> 5];
    if (lane < 9) {
        const int s = lane / 3, d = lane % 3;
        const int i = unit_atom<MOL>(A, u, s);
        const P3MGeom &g = A.g;
        const float h = d == 0 ? g.h.x : (d == 1 ? g.h.y : g.h.z);
        const float lo = d == 0 ? g.lo.x : (d == 1 ? g.lo.y : g.lo.z);
        const int n = d == 0 ? g.sz.x : (d == 1 ? g.sz.y : g.sz.z);
        const float p = (i >= 0 ? reinterpret_cast<const float *>(A.xs)[4 * (size_t)i + d] : lo) - lo;
        const int ng = (int)floorf((p + 0.5f * h) / h);
        float w[5];
        w5(p / h - (float)ng, w);
        float *const ws = d == 0 ? S.wx[s] : (d == 1 ? S.wy[s] : S.wz[s]);
        int *const os = d == 0 ? S.ox[s] : (d == 1 ? S.oy[s] : S.pz[s]);
        const int stride = d == 0 ? g.sz.y * g.sz.z : (d == 1 ? g.sz.z : 1);
#pragma unroll
        for (int c = 0; c < 5; c++) {
            ws[c] = w[c];
            os[c] = wrapi(ng + c - 2, n) * stride;
        }
        if (d == 0) S.q[s] = i >= 0 ? A.qs[i] : 0.f;
    }
    __syncwarp();
    float3 e[3];
#pragma unroll
    for (int s = 0; s < 3; s++) {
        e[s] = make_float3(0.f, 0.f, 0.f);
        if (S.q[s] == 0.f) continue;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int t = 32 * k + lane;
            if (t < 125) {
                const int r = t / 5, c = t % 5, a = r / 5, b = r % 5;
                const float w = S.wx[s][a] * S.wy[s][b] * S.wz[s][c];
                // (the address comes from positions read after the wait, so the
                // load cannot go ahead of it; as a plain load the chain takes
                // 33.2 us for 31.2 at 4,096 molecules, 143 for 135 at 32,768)
                const float4 v = __ldg(A.e4 + (S.ox[s][a] + S.oy[s][b] + S.pz[s][c]));
                e[s].x += w * v.x;
                e[s].y += w * v.y;
                e[s].z += w * v.z;
            }
        }
    }
#pragma unroll
    for (int s = 0; s < 3; s++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            e[s].x += __shfl_xor_sync(0xffffffffu, e[s].x, o);
            e[s].y += __shfl_xor_sync(0xffffffffu, e[s].y, o);
            e[s].z += __shfl_xor_sync(0xffffffffu, e[s].z, o);
        }
    }
    if (MOL && lane == 3 && A.four_site) A.fs[mol_atoms(A, u).x] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (lane >= 3) return;
    const int i = unit_atom<MOL>(A, u, lane);
    const float q = S.q[lane];
    if (i < 0 || (ACC && q == 0.f)) return;
    const float3 m = lane == 0 ? e[0] : (lane == 1 ? e[1] : e[2]);
    const float s = A.g.qunit * q * A.niv;
    float4 f = MOL ? make_float4(0.f, 0.f, 0.f, 0.f) : A.fs[i];
    if (ACC) {
        f.x += s * m.x;
        f.y += s * m.y;
        f.z += s * m.z;
    } else {
        f.x = s * m.x;
        f.y = s * m.y;
        f.z = s * m.z;
    }
    A.fs[i] = f;
}

}  // namespace

FixChargeEwald::FixChargeEwald(State *s, std::string h, std::string g)
    : Fix(s, h, g, "ChargeEwald", FixKind::ChargeEwald) {
    requiresCharges = true;
}

FixChargeEwald::~FixChargeEwald() {
    if (plans) {
        cufftDestroy(plan_r2c);
        cufftDestroy(plan_c2r);
    }
}

int FixChargeEwald::setParameters(int nx, int ny, int nz, double rcut, int ord) {
    auto ok = [](int v) { return v == 32 || v == 64 || v == 128 || v == 256 || v == 512 || v == 1024; };
    if (!ok(nx) || !ok(ny) || !ok(nz)) {
        set_error(MDX_ERR_ARG, "P3M grid %d %d %d: only 2^N sizes 32..1024 are supported (FixChargeEwald.cu:976-987)",
                  nx, ny, nz);
        return MDX_ERR_ARG;
    }
    if (ord != 5) {
        set_error(MDX_ERR_UNSUPPORTED, "P3M interpolation order %d: this library implements order 5", ord);
        return MDX_ERR_UNSUPPORTED;
    }
    sz = make_int3(nx, ny, nz);
    r_cut = rcut;
    order = ord;
    return 0;
}

// total_Q2 (setTotalQ2, :883-914) in FP64 and the secant of :918-967
double FixChargeEwald::findAlpha() {
    State &s = *state;
    double Q2 = 0.0;
    for (auto &a : s.atoms) Q2 += a.q * a.q;
    Q2 *= s.units.qqr_to_eng;
    const double L[3] = {s.box.Ld.x, s.box.Ld.y, s.box.Ld.z};
    const double h[3] = {L[0] / sz.x, L[1] / sz.y, L[2] / sz.z};
    const double nAtoms = (double)s.atoms.size();
    const double rc = r_cut;
    auto dk = [&](double a) {
        double tot = 0.0;
        for (int d = 0; d < 3; d++) {
            double sum = 0.0;
            for (int m = 0; m < order; m++) sum += kAmp[order - 1][m] * std::pow(h[d] * a, 2 * m);
            tot += 1.0 / (L[d] * L[d]) * std::pow(a * h[d], order) * std::sqrt(a * L[d] / nAtoms * std::sqrt(2.0 * M_PI) * sum);
        }
        return Q2 / 3.0 * tot;
    };
    auto dr = [&](double a) { return 2 * Q2 / std::sqrt(nAtoms * rc * L[0] * L[1] * L[2]) * std::exp(-a * a * rc * rc); };
    double xa = 0.0, xb = 4.79853 / rc;
    double ya = dk(xa) - dr(xa), yb = dk(xb) - dr(xb);
    for (int it = 0; it < 100 && std::fabs(yb) / dr(xb) > 1e-5; it++) {
        double kinv = (xb - xa) / (yb - ya);
        ya = yb;
        xa = xb;
        xb = xa - ya * kinv;
        yb = dk(xb) - dr(xb);
    }
    return xb;
}

namespace {
template <int N>
int own_fft_setup();
}  // namespace

int FixChargeEwald::prepareForRun() {
    State &s = *state;
    if (r_cut < 0) r_cut = s.rCut;
    alpha = alpha_user > 0 ? alpha_user : findAlpha();
    const size_t ng = (size_t)sz.x * sz.y * sz.z;
    const size_t nk = (size_t)sz.x * sz.y * (sz.z / 2 + 1);
    if (int e = rho.alloc(ng)) return e;
    if (int e = rho_k.alloc(nk)) return e;
    if (int e = e_k.alloc(3 * nk)) return e;
    if (int e = e_r.alloc(3 * ng)) return e;
    if (int e = green.alloc(nk)) return e;
    if (int e = energy_acc.alloc(1)) return e;
    if (!plans) {
        if (cufftPlan3d(&plan_r2c, sz.x, sz.y, sz.z, CUFFT_R2C) != CUFFT_SUCCESS) {
            set_error(MDX_ERR_CUDA, "cufftPlan3d R2C failed");
            return MDX_ERR_CUDA;
        }
        int dims[3] = {sz.x, sz.y, sz.z};
        if (cufftPlanMany(&plan_c2r, 3, dims, nullptr, 1, (int)nk, nullptr, 1, (int)ng, CUFFT_C2R, 3) !=
            CUFFT_SUCCESS) {
            set_error(MDX_ERR_CUDA, "cufftPlanMany C2R failed");
            return MDX_ERR_CUDA;
        }
        plans = true;
    }
    cufftSetStream(plan_r2c, s.stream);
    cufftSetStream(plan_c2r, s.stream);
    if (int e = f_recip.alloc(std::max(s.gpd.n, 1))) return e;
    // own FFT for cubic 32^3, 64^3 and 128^3 meshes (cuFFT for every other
    // size: two component planes of 256^3 exceed a block's shared memory)
    own_fft = sz.x == sz.y && sz.y == sz.z && (sz.x == 32 || sz.x == 64 || sz.x == 128);
    if (own_fft) {
        if (int e = e4.alloc(ng)) return e;
        if (int e = tw.alloc(sz.x)) return e;
        std::vector<float2> h(sz.x);
        for (int k = 0; k < sz.x; k++)
            h[k] = make_float2((float)std::cos(-2.0 * M_PI * k / sz.x), (float)std::sin(-2.0 * M_PI * k / sz.x));
        MDX_CUDA_TRY(cudaMemcpy(tw.p, h.data(), h.size() * sizeof(float2), cudaMemcpyHostToDevice));
        if (int e = sz.x == 32 ? own_fft_setup<32>() : (sz.x == 64 ? own_fft_setup<64>() : own_fft_setup<128>()))
            return e;
        if (int e = green_own.alloc(nk)) return e;
    }
    // Green function on the half spectrum (Green_function_cu), on the device
    if (int e = computeGreen(s.stream)) return e;
    prepared = true;
    return 0;
}

namespace {
FFTArgs fft_args(State &s, FixChargeEwald &f) {
    FFTArgs A{};
    A.n = f.sz.x;
    A.rho = f.rho.p;
    A.mid1 = f.rho_k.p;
    A.mid2 = f.e_k.p;
    A.e4 = f.e4.p;
    A.green = f.green_own.p;
    A.tw = f.tw.p;
    A.tpl = make_float3((float)(6.28318530717958647693 / s.box.Ld.x), (float)(6.28318530717958647693 / s.box.Ld.y),
                        (float)(6.28318530717958647693 / s.box.Ld.z));
    return A;
}

// What bounds the three kernels is latency, a load, two or four line
// transforms and a store each.  Solve stage (hot, one B200), before -> now:
// 64^3 19.1 -> 11.3 us, 32^3 7.4 -> 6.2 us; 128^3, cuFFT and the E(k) kernel
// before, whole chain with spread and gather 179 -> 134 us at 32,768 molecules
// (there the spread's atomics and the gather's reads are two thirds).
template <int N>
int own_solve(State &s, FixChargeEwald &f, cudaStream_t st) {
    const FFTArgs A = fft_args(s, f);
    cudaError_t err = cudaSuccess;
    launch_solve<N>(
        [&](auto kern, dim3 grid, dim3 block, size_t smem) {
            const cudaError_t e = launch_pdl_prio(true, kern, grid, block, smem, st, A, (const FFTArgs *)nullptr);
            if (e != cudaSuccess) err = e;
        },
        1);
    MDX_CUDA_TRY(err);
    return 0;
}

template <int N>
int own_fft_setup() {
    constexpr int row = N * Line<N>::PITCH * (int)sizeof(float2);
    MDX_CUDA_TRY(cudaFuncSetAttribute(k_fft_zy<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, row));
    MDX_CUDA_TRY(cudaFuncSetAttribute(k_ifft_yz<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * row));
    return 0;
}
}  // namespace

namespace {
// the optimal influence function of order-5 P3M on the half spectrum
// (Green_function_cu, FixChargeEwald.cu:218-294), one thread per k, FP64:
// sum over the aliasing images m within +-lim of the charge assignment
// function's transform W^(2 order) and the reference force R(k_m)
// (green_own, may be null: the same values as (kx, kz, ky), the own FFT's layout)
__global__ void k_green(int3 sz, double3 L, double alpha, int lim, float *__restrict__ green,
                        float *__restrict__ green_own) {
    const int nzh = sz.z / 2 + 1;
    const size_t nk = (size_t)sz.x * sz.y * nzh;
    const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nk) return;
    const int iz = (int)(id % nzh);
    const int iy = (int)((id / nzh) % sz.y);
    const int ix = (int)(id / ((size_t)nzh * sz.y));
    const double tp = 6.28318530717958647693;
    const double h0 = L.x / sz.x, h1 = L.y / sz.y, h2 = L.z / sz.z;
    const double kx = tp * (ix > sz.x / 2 ? ix - sz.x : ix) / L.x;
    const double ky = tp * (iy > sz.y / 2 ? iy - sz.y : iy) / L.y;
    const double kz = tp * iz / L.z;
    const double k2 = kx * kx + ky * ky + kz * kz;
    const double f4a = 0.25 / alpha / alpha;
    double val = 0.0;
    if (k2 != 0.0) {
        double s1 = 0.0, s2 = 0.0;
        for (int mx = -lim; mx <= lim; mx++)
            for (int my = -lim; my <= lim; my++)
                for (int mz = -lim; mz <= lim; mz++) {
                    const double px = kx + tp * mx / h0, py = ky + tp * my / h1, pz = kz + tp * mz / h2;
                    const double pp = px * px + py * py + pz * pz;
                    const double W = sinc(px * h0 * 0.5) * sinc(py * h1 * 0.5) * sinc(pz * h2 * 0.5);
                    const double W2 = W * W, W4 = W2 * W2, W8 = W4 * W4;
                    const double W10 = W8 * W2;  // W^(2 order), order 5
                    s1 += 12.56637061435917295385 * exp(-pp * f4a) * (kx * px + ky * py + kz * pz) / pp * W10;
                    s2 += W10;
                }
        val = s1 / (s2 * s2) / k2;
    }
    green[id] = (float)val;
    if (green_own) green_own[((size_t)ix * nzh + iz) * sz.y + iy] = (float)val;
}
}  // namespace

int FixChargeEwald::computeGreen(cudaStream_t st) {
    State &s = *state;
    const double L[3] = {s.box.Ld.x, s.box.Ld.y, s.box.Ld.z};
    const double h[3] = {L[0] / sz.x, L[1] / sz.y, L[2] / sz.z};
    const int lim = (int)(alpha * std::pow(h[0] * h[1] * h[2], 1.0 / 3.0) / 3.14159 * std::sqrt(-std::log(10E-7))) + 1;
    const size_t nk = (size_t)sz.x * sz.y * (sz.z / 2 + 1);
    k_green<<<(unsigned)((nk + 255) / 256), 256, 0, st>>>(sz, make_double3(L[0], L[1], L[2]), alpha, lim, green.p,
                                                          own_fft ? green_own.p : nullptr);
    MDX_LAUNCHED();
    MDX_CUDA_TRY(cudaGetLastError());
    return 0;
}

// FixChargeEwald::handleBoundsChange (FixChargeEwald.cu:1200-1229): the
// splitting parameter for the new box (unless set by hand) and the Green
// function
int FixChargeEwald::boxChanged() {
    if (!prepared) return 0;
    alpha = alpha_user > 0 ? alpha_user : findAlpha();
    return computeGreen(state->stream);
}

int FixChargeEwald::spread(cudaStream_t st) {
    State &s = *state;
    const size_t ng = (size_t)sz.x * sz.y * sz.z;
    MDX_CUDA_TRY(cudaMemsetAsync(rho.p, 0, ng * sizeof(float), st));
    MDX_CUDA_TRY(launch_pdl_prio(true, k_spread5, dim3((s.gpd.n + 47) / 48), dim3(256), 0, st, p3m_args(s, *this),
                                 (const P3MArgs *)nullptr));
    return 0;
}

int FixChargeEwald::solve(cudaStream_t st) {
    State &s = *state;
    if (own_fft)
        return sz.x == 32 ? own_solve<32>(s, *this, st)
                          : (sz.x == 64 ? own_solve<64>(s, *this, st) : own_solve<128>(s, *this, st));
    const size_t nk = (size_t)sz.x * sz.y * (sz.z / 2 + 1);
    cufftSetStream(plan_r2c, st);
    cufftSetStream(plan_c2r, st);
    if (cufftExecR2C(plan_r2c, rho.p, (cufftComplex *)rho_k.p) != CUFFT_SUCCESS) {
        set_error(MDX_ERR_CUDA, "cufftExecR2C failed");
        return MDX_ERR_CUDA;
    }
    k_efield<<<(unsigned)((nk + 255) / 256), 256, 0, st>>>(p3m_args(s, *this), nullptr);
    MDX_LAUNCHED();
    if (cufftExecC2R(plan_c2r, (cufftComplex *)e_k.p, e_r.p) != CUFFT_SUCCESS) {
        set_error(MDX_ERR_CUDA, "cufftExecC2R failed");
        return MDX_ERR_CUDA;
    }
    return 0;
}

int FixChargeEwald::gather(bool accumulate, cudaStream_t st) {
    State &s = *state;
    const P3MArgs A = p3m_args(s, *this);
    if (own_fft) {
        MDX_CUDA_TRY(launch_pdl_prio(true, accumulate ? k_gather4<false, true> : k_gather4<false, false>,
                                     dim3(mesh_blocks<false>(s.gpd.n, 0)), dim3(kMeshWarps * 32), 0, st, A,
                                     (const P3MArgs *)nullptr));
        return 0;
    }
    if (accumulate)
        k_gather<true><<<(s.gpd.n + 127) / 128, 128, 0, st>>>(A, nullptr);
    else
        k_gather<false><<<(s.gpd.n + 127) / 128, 128, 0, st>>>(A, nullptr);
    MDX_LAUNCHED();
    return 0;
}

int FixChargeEwald::gather_to(float4 *out, cudaStream_t st) {
    State &s = *state;
    P3MArgs A = p3m_args(s, *this);
    A.fs = out;
    if (own_fft) {
        MDX_CUDA_TRY(launch_pdl_prio(true, k_gather4<false, false>, dim3(mesh_blocks<false>(s.gpd.n, 0)),
                                     dim3(kMeshWarps * 32), 0, st, A, (const P3MArgs *)nullptr));
    } else {
        k_gather<false><<<(s.gpd.n + 127) / 128, 128, 0, st>>>(A, nullptr);
        MDX_LAUNCHED();
    }
    return 0;
}

// the molecule form of spread and gather (every atom in a rigid molecule,
// all molecules four-site with uncharged oxygens or all three-site, own FFT)
bool FixChargeEwald::mol_form_ok(const FixRigid &r) const {
    const State &s = *state;
    if (!own_fft || r.mol_ids.empty() || !r.d_mol_idx.p) return false;
    const bool four = r.mol_ids[0].w >= 0;
    size_t members = 0;
    for (const int4 &m : r.mol_ids) {
        if ((m.w >= 0) != four) return false;
        if (four && s.atoms[m.x].q != 0.0) return false;
        members += four ? 4 : 3;
    }
    return members == s.atoms.size();
}

P3MArgs mol_args(State &s, FixChargeEwald &f, const FixRigid &r) {
    P3MArgs A = p3m_args(s, f);
    A.mol_idx = r.d_mol_idx.p;
    A.nmol = (int)r.mol_ids.size();
    A.four_site = r.mol_ids[0].w >= 0 ? 1 : 0;
    A.slots = s.mf.on ? 1 : 0;
    return A;
}

int FixChargeEwald::spread_mol(cudaStream_t st, const FixRigid &r) {
    State &s = *state;
    const size_t ng = (size_t)sz.x * sz.y * sz.z;
    MDX_CUDA_TRY(cudaMemsetAsync(rho.p, 0, ng * sizeof(float), st));
    const P3MArgs A = mol_args(s, *this, r);
    const int warps = (A.nmol + 1) / 2;
    // two-warp blocks: they slot in beside the pair kernel's (measured +1 % per
    // water step against 256-thread blocks)
    MDX_CUDA_TRY(launch_pdl_prio(true, k_spread_mol, dim3((warps + 1) / 2), dim3(64), 0, st, A,
                                 (const P3MArgs *)nullptr));
    return 0;
}

int FixChargeEwald::gather_mol_to(float4 *out, cudaStream_t st, const FixRigid &r) {
    State &s = *state;
    P3MArgs A = mol_args(s, *this, r);
    A.fs = out;
    MDX_CUDA_TRY(launch_pdl_prio(true, k_gather4<true, false>, dim3(mesh_blocks<true>(0, A.nmol)),
                                 dim3(kMeshWarps * 32), 0, st, A, (const P3MArgs *)nullptr));
    return 0;
}

int FixChargeEwald::compute(int virialMode) {
    State &s = *state;
    if (int e = spread(s.stream)) return e;
    if (int e = solve(s.stream)) return e;
    if (int e = gather(true, s.stream)) return e;
    return virialMode ? ewald_recip_virial(s, *this) : 0;
}

// the reciprocal-space virial (FixChargeEwald::compute with virialMode,
// FixChargeEwald.cu:1455-1466): spread, R2C, k-space sum, onto atom 0
int ewald_recip_virial(State &s, FixChargeEwald &f) {
    if (int e = f.spread(s.stream)) return e;
    cufftSetStream(f.plan_r2c, s.stream);
    if (cufftExecR2C(f.plan_r2c, f.rho.p, (cufftComplex *)f.rho_k.p) != CUFFT_SUCCESS) {
        set_error(MDX_ERR_CUDA, "cufftExecR2C failed");
        return MDX_ERR_CUDA;
    }
    if (int e = f.vir_acc.alloc(6)) return e;
    MDX_CUDA_TRY(cudaMemsetAsync(f.vir_acc.p, 0, 6 * sizeof(double), s.stream));
    const size_t nk = (size_t)f.sz.x * f.sz.y * (f.sz.z / 2 + 1);
    const double3 tpl = make_double3(2.0 * M_PI / s.box.Ld.x, 2.0 * M_PI / s.box.Ld.y, 2.0 * M_PI / s.box.Ld.z);
    k_recip_virial<<<148, 256, 0, s.stream>>>(f.sz, f.rho_k.p, f.green.p, nk, tpl, f.alpha, f.vir_acc.p);
    MDX_LAUNCHED();
    const double V = s.box.Ld.x * s.box.Ld.y * s.box.Ld.z;
    k_add_field_virial<<<1, 32, 0, s.stream>>>(s.gpd.virials.p, f.vir_acc.p, 0.5 / V);
    MDX_LAUNCHED();
    return 0;
}

int ewald_recip_energy(State &s, FixChargeEwald &f, double *out) {
    if (int e = f.spread(s.stream)) return e;
    cufftSetStream(f.plan_r2c, s.stream);
    if (cufftExecR2C(f.plan_r2c, f.rho.p, (cufftComplex *)f.rho_k.p) != CUFFT_SUCCESS) {
        set_error(MDX_ERR_CUDA, "cufftExecR2C failed");
        return MDX_ERR_CUDA;
    }
    const size_t nk = (size_t)f.sz.x * f.sz.y * (f.sz.z / 2 + 1);
    MDX_CUDA_TRY(cudaMemsetAsync(f.energy_acc.p, 0, sizeof(double), s.stream));
    k_recip_energy<<<148, 256, 0, s.stream>>>(f.sz, f.rho_k.p, f.green.p, nk, f.energy_acc.p);
    MDX_LAUNCHED();
    double sumG = 0.0;
    MDX_CUDA_TRY(cudaMemcpyAsync(&sumG, f.energy_acc.p, sizeof(double), cudaMemcpyDeviceToHost, s.stream));
    MDX_CUDA_TRY(cudaStreamSynchronize(s.stream));
    double Q2 = 0.0;
    for (auto &a : s.atoms) Q2 += a.q * a.q;
    Q2 *= s.units.qqr_to_eng;
    const double V = s.box.Ld.x * s.box.Ld.y * s.box.Ld.z;
    *out = 0.5 * sumG / V - f.alpha / std::sqrt(M_PI) * Q2;
    return 0;
}

// ---- batched replicas -------------------------------------------------------
// Replicas are grouped by mesh size; each class gets contiguous pools that its
// replicas' buffers view, so a batched cuFFT plan per class covers them all.
// Spread, E(k) and gather are one launch each for every replica.
int batch_p3m_prepare(Batch &b) {
    const int R = (int)b.reps.size();
    for (int r = 0; r < R; r++) {
        FixChargeEwald *f = b.reps[r]->ewaldFix();
        Batch::FFTClass *c = nullptr;
        for (auto &k : b.fft)
            if (k->sz.x == f->sz.x && k->sz.y == f->sz.y && k->sz.z == f->sz.z) c = k.get();
        if (!c) {
            b.fft.emplace_back(new Batch::FFTClass());
            c = b.fft.back().get();
            c->sz = f->sz;
        }
        c->reps.push_back(r);
    }
    for (auto &cp : b.fft) {
        Batch::FFTClass &c = *cp;
        const int K = (int)c.reps.size();
        const size_t ng = (size_t)c.sz.x * c.sz.y * c.sz.z;
        const size_t nk = (size_t)c.sz.x * c.sz.y * (c.sz.z / 2 + 1);
        if (int e = c.rho.alloc(K * ng)) return e;
        if (int e = c.rho_k.alloc(K * nk)) return e;
        if (int e = c.e_k.alloc(K * 3 * nk)) return e;
        if (int e = c.e_r.alloc(K * 3 * ng)) return e;
        for (int j = 0; j < K; j++) {
            FixChargeEwald *f = b.reps[c.reps[j]]->ewaldFix();
            f->rho.view(c.rho.p + j * ng, ng, cp);
            f->rho_k.view(c.rho_k.p + j * nk, nk, cp);
            f->e_k.view(c.e_k.p + j * 3 * nk, 3 * nk, cp);
            f->e_r.view(c.e_r.p + j * 3 * ng, 3 * ng, cp);
            b.reps[c.reps[j]]->box_gen++;  // graphs captured so far hold the addresses before
        }
        c.own = true;
        for (int j = 0; j < K; j++) c.own = c.own && b.reps[c.reps[j]]->ewaldFix()->own_fft;
        if (c.own) {
            std::vector<FFTArgs> ft(K);
            for (int j = 0; j < K; j++) ft[j] = fft_args(*b.reps[c.reps[j]], *b.reps[c.reps[j]]->ewaldFix());
            if (int e = c.tab.alloc(K * sizeof(FFTArgs))) return e;
            MDX_CUDA_TRY(cudaMemcpy(c.tab.p, ft.data(), K * sizeof(FFTArgs), cudaMemcpyHostToDevice));
        } else {
            int dims[3] = {c.sz.x, c.sz.y, c.sz.z};
            if (cufftPlanMany(&c.r2c, 3, dims, nullptr, 1, (int)ng, nullptr, 1, (int)nk, CUFFT_R2C, K) !=
                    CUFFT_SUCCESS ||
                cufftPlanMany(&c.c2r, 3, dims, nullptr, 1, (int)nk, nullptr, 1, (int)ng, CUFFT_C2R, 3 * K) !=
                    CUFFT_SUCCESS) {
                set_error(MDX_ERR_CUDA, "batched cufftPlanMany failed");
                return MDX_ERR_CUDA;
            }
        }
    }
    b.p3m_own = true;
    for (auto &cp : b.fft) b.p3m_own = b.p3m_own && cp->own;
    std::vector<P3MArgs> h(R);
    for (int r = 0; r < R; r++) h[r] = p3m_args(*b.reps[r], *b.reps[r]->ewaldFix());
    if (int e = b.tab_p3m.alloc(R * sizeof(P3MArgs))) return e;
    MDX_CUDA_TRY(cudaMemcpy(b.tab_p3m.p, h.data(), R * sizeof(P3MArgs), cudaMemcpyHostToDevice));
    if (!b.p3m_own)
        for (auto &cp : b.fft) {
            const int K = (int)cp->reps.size();
            std::vector<P3MArgs> hc(K);
            cp->max_n = 0;
            for (int j = 0; j < K; j++) {
                hc[j] = h[cp->reps[j]];
                cp->max_n = std::max(cp->max_n, hc[j].n);
            }
            if (int e = cp->p3m.alloc(K * sizeof(P3MArgs))) return e;
            MDX_CUDA_TRY(cudaMemcpy(cp->p3m.p, hc.data(), K * sizeof(P3MArgs), cudaMemcpyHostToDevice));
        }
    // the molecule form of spread and gather, as the single system's fused
    // step: the charged sites of each molecule only, the reciprocal forces
    // stored into each replica's per-step buffer by the P3M branch itself
    b.p3m_mol = b.p3m_own;
    for (State *s : b.reps) b.p3m_mol = b.p3m_mol && s->ewaldFix()->mol_form_ok(*s->rigidFix());
    if (b.p3m_mol) {
        for (int r = 0; r < R; r++) {
            State &s = *b.reps[r];
            h[r] = mol_args(s, *s.ewaldFix(), *s.rigidFix());
            h[r].fs = s.ewaldFix()->f_recip.p;
        }
        if (int e = b.tab_p3m_mol.alloc(R * sizeof(P3MArgs))) return e;
        MDX_CUDA_TRY(cudaMemcpy(b.tab_p3m_mol.p, h.data(), R * sizeof(P3MArgs), cudaMemcpyHostToDevice));
    }
    return 0;
}

int batch_p3m_spread_solve(Batch &b, cudaStream_t st) {
    const unsigned R = (unsigned)b.reps.size();
    const P3MArgs *tab = reinterpret_cast<const P3MArgs *>(b.tab_p3m.p);
    P3MArgs A = p3m_args(*b.reps[0], *b.reps[0]->ewaldFix());  // sizing only
    A.n = b.max_n;
    for (auto &c : b.fft) MDX_CUDA_TRY(cudaMemsetAsync(c->rho.p, 0, c->rho.n * sizeof(float), st));
    if (b.p3m_mol) {
        const int warps = (b.max_mol + 1) / 2;
        k_spread_mol<<<dim3((warps + 1) / 2, R), 64, 0, st>>>(A, reinterpret_cast<const P3MArgs *>(b.tab_p3m_mol.p));
    } else {
        k_spread5<<<dim3((A.n + 47) / 48, R), 256, 0, st>>>(A, tab);
    }
    MDX_LAUNCHED();
    // each mesh class by itself: the three FFT kernels of the single system
    // over the class's replicas, or batched cuFFT around the E(k) kernel where
    // the own FFT does not serve the mesh
    for (auto &c : b.fft) {
        const unsigned K = (unsigned)c->reps.size();
        if (c->own) {
            const FFTArgs a0 = fft_args(*b.reps[c->reps[0]], *b.reps[c->reps[0]]->ewaldFix());
            const FFTArgs *ft = reinterpret_cast<const FFTArgs *>(c->tab.p);
            auto launch = [&](auto kern, dim3 grid, dim3 block, size_t smem) {
                kern<<<grid, block, smem, st>>>(a0, ft);
            };
            if (c->sz.x == 32) launch_solve<32>(launch, K);
            else if (c->sz.x == 64) launch_solve<64>(launch, K);
            else launch_solve<128>(launch, K);
            g_launches += 3;
            continue;
        }
        cufftSetStream(c->r2c, st);
        if (cufftExecR2C(c->r2c, c->rho.p, (cufftComplex *)c->rho_k.p) != CUFFT_SUCCESS) {
            set_error(MDX_ERR_CUDA, "batched cufftExecR2C failed");
            return MDX_ERR_CUDA;
        }
        const size_t nk = (size_t)c->sz.x * c->sz.y * (c->sz.z / 2 + 1);
        k_efield<<<dim3((unsigned)((nk + 255) / 256), K), 256, 0, st>>>(A,
                                                                        reinterpret_cast<const P3MArgs *>(c->p3m.p));
        MDX_LAUNCHED();
        cufftSetStream(c->c2r, st);
        if (cufftExecC2R(c->c2r, (cufftComplex *)c->e_k.p, c->e_r.p) != CUFFT_SUCCESS) {
            set_error(MDX_ERR_CUDA, "batched cufftExecC2R failed");
            return MDX_ERR_CUDA;
        }
    }
    MDX_CUDA_TRY(cudaGetLastError());
    return 0;
}

int batch_p3m_gather(Batch &b, cudaStream_t st) {
    const P3MArgs *tab = reinterpret_cast<const P3MArgs *>(b.tab_p3m.p);
    P3MArgs A = p3m_args(*b.reps[0], *b.reps[0]->ewaldFix());
    A.n = b.max_n;
    if (b.p3m_mol) {  // into each replica's per-step buffer (the second half adds it)
        k_gather4<true, false><<<dim3(mesh_blocks<true>(0, b.max_mol), (unsigned)b.reps.size()), kMeshWarps * 32, 0,
                                 st>>>(A, reinterpret_cast<const P3MArgs *>(b.tab_p3m_mol.p));
        MDX_LAUNCHED();
        return 0;
    }
    if (b.p3m_own) {
        k_gather4<false, true><<<dim3(mesh_blocks<false>(A.n, 0), (unsigned)b.reps.size()), kMeshWarps * 32, 0, st>>>(
            A, tab);
        MDX_LAUNCHED();
        return 0;
    }
    for (auto &c : b.fft) {
        const unsigned K = (unsigned)c->reps.size();
        const P3MArgs *ct = reinterpret_cast<const P3MArgs *>(c->p3m.p);
        if (c->own)
            k_gather4<false, true><<<dim3(mesh_blocks<false>(c->max_n, 0), K), kMeshWarps * 32, 0, st>>>(A, ct);
        else
            k_gather<true><<<dim3((c->max_n + 127) / 128, K), 128, 0, st>>>(A, ct);
        MDX_LAUNCHED();
    }
    return 0;
}

}  // namespace mdx
