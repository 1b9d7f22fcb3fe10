// Kernels of the warm-start network: periodic 3-D convolutions (BF16 weights, FP32 activations
// and accumulation), GELU, bias and loss reductions, Adam.
//
// Layouts.  A volume of C channels on a d x h x w grid is [C][z][y][x] with x fastest,
// the point order of the solver's xi(no, nx, ny, nz) with io dropped.  Weights of a
// convolution are [cout][cin][kz][ky][kx]; weights of the transposed (up-sampling)
// convolution are [cin][cout][kz][ky][kx] (the coarse channel first).
//
// Three convolution kinds, all periodic like the solver's box:
//   KS=3, S=1: 3x3x3, wrap-around padding of one voxel;
//   KS=2, S=2: 2x2x2 stride 2 (down-sampling), and its transpose (up-sampling);
//   KS=1, S=1: pointwise (the output head).
// The first kind has kernels on the matrix instructions (k_conv3, k_conv3_wgrad); the others, a
// quarter of the time, gather-GEMMs on FP32 CUDA cores, k_conv_gemm<MODE,...>: a 64-voxel x
// 32-channel output tile per CTA, reduction chunks of 32 staged in shared memory (A gathered from
// the activation volume, B from the weights, converted to FP32).
#pragma once

#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "common.cuh"

namespace mdft {
namespace wn {

struct Vol {
    int d, h, w;
    __host__ __device__ long long n() const { return (long long)d * h * w; }
};

constexpr int kBM = 64;   // voxels per tile
constexpr int kBN = 32;   // channels per tile
constexpr int kBK = 32;   // reduction chunk
constexpr int kThreads = 256;

enum ConvMode {
    kFwd = 0,     // Y[co][o] = sum_{ci,k} W[co][ci][k] X[ci][o*S + k]               (conv forward)
    kBwdData = 1, // dX[ci][i] = sum_{co,k} W[co][ci][k] dY[co][i - k]              (KS = 1 only)
    kParity = 2,  // F[cf][2o+a] = sum_cc W[cc][cf][a] C[cc][o]                      (KS = 2, S = 2:
                  //  the transposed convolution, and the data gradient of the stride-2 conv)
};

struct ConvArgs {
    const float *x;            // gathered operand (kFwd: input X; kBwdData: dY; kParity: coarse C)
    const __nv_bfloat16 *wt;   // weights
    const float *bias;         // per output channel, or null
    float *y;                  // output volume
    int cin, cout;             // channels of the gathered operand / of the output
    Vol vin, vout;             // grid of the gathered operand / of the output
    int accumulate;            // 1: y += result, 0: y = result
};

// One output tile.  blockIdx.x: voxel tile, blockIdx.y: channel tile, blockIdx.z: parity
// class a = (az*2 + ay)*2 + ax (kParity only).
template <int MODE, int KS, int S>
__global__ void __launch_bounds__(kThreads) k_conv_gemm(ConvArgs a) {
    constexpr int K3 = KS * KS * KS;
    __shared__ float As[kBK][kBM];
    __shared__ __align__(16) float Bs[kBK][kBN + 4];
    const int tid = threadIdx.x;
    const int v = tid & (kBM - 1);     // this thread's voxel in the tile
    const int cg = tid >> 6;           // its group of 8 output channels
    const int co0 = blockIdx.y * kBN;
    const int par = MODE == kParity ? (int)blockIdx.z : 0;
    // voxels are enumerated over the grid the reduction is gathered on: the output grid
    // for kFwd / kBwdData, the coarse grid for kParity
    const Vol vg = MODE == kParity ? a.vin : a.vout;
    const long long nv = vg.n();
    const long long o = (long long)blockIdx.x * kBM + v;
    const bool live = o < nv;
    int ox = 0, oy = 0, oz = 0;
    if (live) {
        ox = (int)(o % vg.w);
        long long t = o / vg.w;
        oy = (int)(t % vg.h);
        oz = (int)(t / vg.h);
    }
    // reduction length: kFwd cin*K3, kBwdData cin*K3 (cin = channels of dY), kParity cin
    const int Ktot = MODE == kParity ? a.cin : a.cin * K3;
    const long long nin = a.vin.n();
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (int k0 = 0; k0 < Ktot; k0 += kBK) {
        // A: this thread's voxel, reduction rows (tid >> 6) + 4 j
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int kr = cg + 4 * j;
            const int kk = k0 + kr;
            float val = 0.f;
            if (live && kk < Ktot) {
                if (MODE == kParity) {
                    val = a.x[(long long)kk * nin + o];
                } else {
                    const int c = kk / K3, kof = kk - c * K3;
                    const int kx = kof % KS, ky = (kof / KS) % KS, kz = kof / (KS * KS);
                    const int ix = ox * S + kx, iy = oy * S + ky, iz = oz * S + kz;
                    val = a.x[(long long)c * nin + ((long long)iz * a.vin.h + iy) * a.vin.w + ix];
                }
            }
            As[kr][v] = val;
        }
        // B: rows of the weights, (channel c, reduction kk) -> Bs[kk][c]
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int e = tid + kThreads * j;
            const int c = e >> 5, kr = e & 31;
            const int co = co0 + c, kk = k0 + kr;
            float val = 0.f;
            if (co < a.cout && kk < Ktot) {
                long long wi;
                if (MODE == kFwd) {
                    wi = (long long)co * Ktot + kk;                           // W[co][ci][k]
                } else if (MODE == kBwdData) {
                    const int cc = kk / K3, kof = kk - cc * K3;               // W[cc][co][k]
                    wi = ((long long)cc * a.cout + co) * K3 + kof;
                } else {
                    wi = ((long long)kk * a.cout + co) * 8 + par;             // W[kk][co][a]
                }
                val = __bfloat162float(a.wt[wi]);
            }
            Bs[kr][c] = val;
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < kBK; ++k) {
            const float av = As[k][v];
            const float4 b0 = *reinterpret_cast<const float4 *>(&Bs[k][cg * 8]);
            const float4 b1 = *reinterpret_cast<const float4 *>(&Bs[k][cg * 8 + 4]);
            acc[0] = fmaf(av, b0.x, acc[0]); acc[1] = fmaf(av, b0.y, acc[1]);
            acc[2] = fmaf(av, b0.z, acc[2]); acc[3] = fmaf(av, b0.w, acc[3]);
            acc[4] = fmaf(av, b1.x, acc[4]); acc[5] = fmaf(av, b1.y, acc[5]);
            acc[6] = fmaf(av, b1.z, acc[6]); acc[7] = fmaf(av, b1.w, acc[7]);
        }
        __syncthreads();
    }
    if (!live) return;
    long long oi = o;
    if (MODE == kParity) {
        const int ax = par & 1, ay = (par >> 1) & 1, az = par >> 2;
        oi = ((long long)(2 * oz + az) * a.vout.h + (2 * oy + ay)) * a.vout.w + (2 * ox + ax);
    }
    const long long nout = a.vout.n();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int co = co0 + cg * 8 + j;
        if (co >= a.cout) break;
        float r = acc[j];
        if (a.bias) r += a.bias[co];
        float *dst = a.y + (long long)co * nout + oi;
        *dst = a.accumulate ? *dst + r : r;
    }
}

struct WgradArgs {
    const float *dy;   // [cout][nout]: gradient at the conv output (coarse for KS=2)
    const float *x;    // [cin][nin]: the conv input
    float *part;       // [nsplit][cout][cin*K3]
    int cin, cout;
    Vol vin, vout;
    long long per_split;  // output voxels per split (a multiple of kBK)
};

// dW[co][ci][k] = sum_o dY[co][o] X[ci][o*S + k]: a 32-channel x 64-column tile per CTA
// over one split of the output voxels (blockIdx.z), partial sums to part[split].
template <int KS, int S>
__global__ void __launch_bounds__(kThreads) k_conv_wgrad(WgradArgs a) {
    constexpr int K3 = KS * KS * KS;
    __shared__ __align__(16) float As[kBK][kBN + 4];  // [voxel][co]
    __shared__ float Bs[kBK][kBM];                    // [voxel][column]
    const int tid = threadIdx.x;
    const int col = tid & (kBM - 1);
    const int cg = tid >> 6;
    const int Ktot = a.cin * K3;
    const int kk = blockIdx.x * kBM + col;  // this thread's weight column
    const bool colok = kk < Ktot;
    int ci = 0, kx = 0, ky = 0, kz = 0;
    if (colok) {
        ci = kk / K3;
        const int kof = kk - ci * K3;
        kx = kof % KS; ky = (kof / KS) % KS; kz = kof / (KS * KS);
    }
    const int co0 = blockIdx.y * kBN;
    const long long nout = a.vout.n(), nin = a.vin.n();
    const long long s0 = (long long)blockIdx.z * a.per_split;
    const long long s1 = s0 + a.per_split < nout ? s0 + a.per_split : nout;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (long long o0 = s0; o0 < s1; o0 += kBK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // dY rows: (co, voxel) -> As[voxel][co]
            const int e = tid + kThreads * j;
            const int c = e >> 5, vv = e & 31;
            const long long o = o0 + vv;
            const int co = co0 + c;
            As[vv][c] = (co < a.cout && o < s1) ? a.dy[(long long)co * nout + o] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {  // X gathered at this column's offset
            const int vv = cg + 4 * j;
            const long long o = o0 + vv;
            float val = 0.f;
            if (colok && o < s1) {
                const int ox = (int)(o % a.vout.w);
                const long long t = o / a.vout.w;
                const int oy = (int)(t % a.vout.h), oz = (int)(t / a.vout.h);
                const int ix = ox * S + kx, iy = oy * S + ky, iz = oz * S + kz;
                val = a.x[(long long)ci * nin + ((long long)iz * a.vin.h + iy) * a.vin.w + ix];
            }
            Bs[vv][col] = val;
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < kBK; ++k) {
            const float bv = Bs[k][col];
            const float4 a0 = *reinterpret_cast<const float4 *>(&As[k][cg * 8]);
            const float4 a1 = *reinterpret_cast<const float4 *>(&As[k][cg * 8 + 4]);
            acc[0] = fmaf(a0.x, bv, acc[0]); acc[1] = fmaf(a0.y, bv, acc[1]);
            acc[2] = fmaf(a0.z, bv, acc[2]); acc[3] = fmaf(a0.w, bv, acc[3]);
            acc[4] = fmaf(a1.x, bv, acc[4]); acc[5] = fmaf(a1.y, bv, acc[5]);
            acc[6] = fmaf(a1.z, bv, acc[6]); acc[7] = fmaf(a1.w, bv, acc[7]);
        }
        __syncthreads();
    }
    if (!colok) return;
    float *dst = a.part + (long long)blockIdx.z * a.cout * Ktot;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int co = co0 + cg * 8 + j;
        if (co >= a.cout) break;
        dst[(long long)co * Ktot + kk] = acc[j];
    }
}

// g[i] (+)= sum over splits of part[s][i]: eight groups of splits per value, each in
// order, in FP64 (the sums cancel: a gradient's terms are much larger than it)
__global__ void __launch_bounds__(256) k_wgrad_reduce(const float *__restrict__ part, float *__restrict__ g, int nsplit, long long n, int accumulate) {
    __shared__ double red[8][32];
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
    const long long i = (long long)blockIdx.x * 32 + lane;
    double s = 0.0;
    if (i < n)
        for (int k = grp; k < nsplit; k += 8) s += part[(long long)k * n + i];
    red[grp][lane] = s;
    __syncthreads();
    if (grp == 0 && i < n) {
        for (int k = 1; k < 8; ++k) s += red[k][lane];
        g[i] = accumulate ? g[i] + (float)s : (float)s;
    }
}

__device__ __forceinline__ float gelu_f(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
    return 0.5f * (1.f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// ---- 3 x 3 x 3 convolutions on the matrix instructions (mma.sync m16n8k16 bf16) ----
//
// A CTA takes an 8 x 4 x 4 tile of voxels and 16 channels; the input tile with its halo (10 x 6 x 6,
// periodic) is staged once per 16 channels and read at the 27 offsets, where the gather-GEMM
// above fetched and indexed every (voxel, tap) anew.  An FP32 operand is staged as three BF16 terms
// of 8 bits each, which is exact; BF16 weights are exact, so a forward or data-gradient product is
// three instructions, a weight gradient's (both sides FP32) six: of the nine products of terms
// those above 2^-24.  The matrix instruction truncates what it accumulates, so each block of 16 of the
// reduction starts from zero, the leading products (16 bits) apart from the smaller ones and, where
// a result goes on through further layers, in two halves, and is added in FP32.  At 48^3 (us,
// gather-GEMM and now): 16 -> 16 channels forward 161 -> 53, data gradient 232 -> 55, weight gradient
// 315 -> 57; 128 -> 128 at 6^3 231 -> 22, 265 -> 18.  Bound by latency: matrix pipe 10 to 35 % busy,
// the fragments' shared-memory reads 15 to 40 %, issue 15 to 45 %.  One pass of the network, forward
// and backward, 4.69 -> 1.86 ms, and its gradients' error against 64 bits on
// random inputs 3.3e-7 -> 2.3e-7 (all products in one accumulator: above 5e-7; the leading ones in
// one block of 16: 3.5e-7).
constexpr int kCX = 8, kCY = 4, kCZ = 4;              // voxel tile
constexpr int kHX = kCX + 2, kHY = kCY + 2, kHZ = kCZ + 2;
constexpr int kHalo = kHX * kHY * kHZ;                // 360: channel pairs t, t + 1, ... are 8 banks apart
constexpr int kC3N = 16;                              // channels of the output per CTA
constexpr int kZPair = 2 * kHX * kHY;                 // a word of the weight gradient holds voxels z, z + 2
constexpr int kPairs = (kHZ - 2) * kHX * kHY;         // 240
constexpr int kPairRow = kPairs + 4, kDyRow = kCX * kCY * 2 + 4;  // rows of 244 and 68: 20 and 4 banks

// x = h + m + l exactly, each the upper half of a float; an infinity is all in h
__device__ __forceinline__ void split3(float x, uint32_t &h, uint32_t &m, uint32_t &l) {
    h = __float_as_uint(x) & 0xFFFF0000u;
    const float r = x == __uint_as_float(h) ? 0.f : x - __uint_as_float(h);
    m = __float_as_uint(r) & 0xFFFF0000u;
    l = __float_as_uint(r - __uint_as_float(m));
}
// the upper halves of a (low) and b (high)
__device__ __forceinline__ uint32_t pack_hi(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }
struct Split3 {
    uint32_t h, m, l;
    __device__ __forceinline__ Split3(float a, float b) {
        uint32_t ah, am, al, bh, bm, bl;
        split3(a, ah, am, al);
        split3(b, bh, bm, bl);
        h = pack_hi(ah, bh);
        m = pack_hi(am, bm);
        l = pack_hi(al, bl);
    }
};
// d = a b + c
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ void mma_bf16_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, const float (&c)[4]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(b0), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
struct Tile3 {
    int x0, y0, z0;
    __device__ __forceinline__ Tile3(int i, const Vol &v) {
        const int nx = (v.w + kCX - 1) / kCX, ny = (v.h + kCY - 1) / kCY;
        x0 = i % nx * kCX;
        y0 = i / nx % ny * kCY;
        z0 = i / nx / ny * kCZ;
    }
};
__host__ __device__ inline int conv3_tiles(const Vol &v) {
    return ((v.w + kCX - 1) / kCX) * ((v.h + kCY - 1) / kCY) * ((v.d + kCZ - 1) / kCZ);
}
// the offset of halo point r of a tile, wrapped
__device__ __forceinline__ int halo_offset(int r, const Tile3 &t, const Vol &v) {
    const int hx = r % kHX, hy = r / kHX % kHY, hz = r / (kHX * kHY);
    int x = t.x0 + hx - 1, y = t.y0 + hy - 1, z = t.z0 + hz - 1;
    x = x < 0 ? x + v.w : x % v.w;
    y = y < 0 ? y + v.h : y % v.h;
    z = z < 0 ? z + v.d : z % v.d;
    return (z * v.h + y) * v.w + x;
}
// Y[co][o] = sum_{ci,k} W[co][ci][k] X[ci][o + k - 1] (BWD = false), or the data gradient
// dX[ci][i] = sum_{co,k} W[co][ci][k] dY[co][i + 1 - k] (BWD: a.cin the channels of dY, a.cout
// those of dX).  act (may be null): also GELU of the result.
// The blocks of a cluster (grid.z) share the input channels, and each finishes a part of the sums:
// the 128 channels at 6^3 voxels are otherwise 32 blocks with a chain of eight stages (80 us; 8
// blocks a cluster: 21).
template <bool BWD>
__global__ void __launch_bounds__(kThreads) k_conv3(ConvArgs a, float *__restrict__ act) {
    __shared__ uint32_t xs[3][8][kHalo];     // [term][channel pair][voxel]
    __shared__ uint32_t ws[27 * 8 * kC3N];   // [tap][channel pair][output channel, ^ 8 for pairs 2, 3 mod 4]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const Vol v = a.vout;
    const Tile3 tl(blockIdx.x, v);
    const int co0 = blockIdx.y * kC3N;
    const long long n = v.n();
    int off[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) off[q] = tid + kThreads * q < kHalo ? halo_offset(tid + kThreads * q, tl, v) : 0;
    const int tz = warp >> 1, ty = (warp & 1) * 2;
    float acc[2][4] = {}, low[2][4] = {};
    const float zero[4] = {0.f, 0.f, 0.f, 0.f};
    const unsigned short *W = reinterpret_cast<const unsigned short *>(a.wt);
    const int rank = blockIdx.z, nrank = gridDim.z;
    for (int c0 = 16 * rank; c0 < a.cin; c0 += 16 * nrank) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int r = tid + kThreads * q;
            if (r >= kHalo) break;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float f[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) f[c] = c0 + 8 * half + c < a.cin ? a.x[(c0 + 8 * half + c) * n + off[q]] : 0.f;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const Split3 sp(f[2 * c], f[2 * c + 1]);
                    xs[0][4 * half + c][r] = sp.h;
                    xs[1][4 * half + c][r] = sp.m;
                    xs[2][4 * half + c][r] = sp.l;
                }
            }
        }
        for (int e = tid; e < 27 * 8 * kC3N; e += kThreads) {
            const int co = co0 + (e & 15), p = e >> 4 & 7, tap = e >> 7, wt = BWD ? 26 - tap : tap;
            uint32_t w2 = 0;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int ci = c0 + 2 * p + q;
                if (ci < a.cin && co < a.cout) w2 |= (uint32_t)W[(BWD ? (long long)ci * a.cout + co : (long long)co * a.cin + ci) * 27 + wt] << (16 * q);
            }
            ws[e ^ (p & 2) << 2] = w2;
        }
        __syncthreads();
#pragma unroll 1
        for (int kz = 0; kz < 3; ++kz)
#pragma unroll
            for (int ky = 0; ky < 3; ++ky)
#pragma unroll
                for (int kx = 0; kx < 3; ++kx) {
                    const int o = ((tz + kz) * kHY + ty + ky) * kHX + g + kx;
                    uint32_t f[3][4];
#pragma unroll
                    for (int k = 0; k < 3; ++k)
#pragma unroll
                        for (int i = 0; i < 4; ++i) f[k][i] = xs[k][t + 4 * (i >> 1)][o + kHX * (i & 1)];
                    const uint32_t *w = ws + ((kz * 3 + ky) * 3 + kx) * 8 * kC3N + t * kC3N;
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int col = (g + 8 * j) ^ (t & 2) << 2;
                        const uint32_t b0 = w[col], b1 = w[4 * kC3N + col];
                        float s[4], u[4];
                        float u2[4];
                        mma_bf16_k8(u, f[0][0], f[0][1], b0, zero);
                        mma_bf16_k8(u2, f[0][2], f[0][3], b1, zero);
                        mma_bf16(s, f[2], b0, b1, zero);
                        mma_bf16(s, f[1], b0, b1, s);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            acc[j][i] += u[i];
                            acc[j][i] += u2[i];
                            low[j][i] += s[i];
                        }
                    }
                }
        __syncthreads();
    }
    float *part = reinterpret_cast<float *>(xs);  // [value][thread]
    if (nrank > 1) {
        for (int k = 0; k < 8; ++k) part[k * kThreads + tid] = acc[k >> 2][k & 3] + low[k >> 2][k & 3];
        cooperative_groups::this_cluster().sync();
    }
    const int x = tl.x0 + g, z = tl.z0 + tz;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if ((4 * j + i) * nrank / 8 != rank) continue;
            const int y = tl.y0 + ty + (i >> 1), co = co0 + 8 * j + 2 * t + (i & 1);
            if (x >= v.w || y >= v.h || z >= v.d || co >= a.cout) continue;
            const long long o = co * n + ((long long)z * v.h + y) * v.w + x;
            float r = acc[j][i] + low[j][i];
            if (nrank > 1) {
                r = 0.f;
                for (int k = 0; k < nrank; ++k) r += cooperative_groups::this_cluster().map_shared_rank(part, k)[(4 * j + i) * kThreads + tid];
            }
            if (a.bias) r += a.bias[co];
            if (a.accumulate) r += a.y[o];
            a.y[o] = r;
            if (act) act[o] = gelu_f(r);
        }
    if (nrank > 1) cooperative_groups::this_cluster().sync();  // the partial sums have been read
}

// dW[co][ci][k] = sum_o dY[co][o] X[ci][o + k - 1]: 16 x 8 channels and every tap per CTA, over
// the voxel tiles of one split (a.per_split of them); a warp has the taps warp, warp + 8, ...
__global__ void __launch_bounds__(kThreads) k_conv3_wgrad(WgradArgs a) {
    __shared__ uint32_t xs[3][8][kPairRow];     // [term][channel][voxels z, z + 2 of the halo]
    __shared__ uint32_t ds[3][kC3N][kDyRow];    // [term][channel][voxels z, z + 2]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const Vol v = a.vout;
    const long long n = v.n();
    const int ci0 = blockIdx.x * 8, co0 = blockIdx.y * kC3N;
    const int t0 = blockIdx.z * (int)a.per_split, t1 = min(t0 + (int)a.per_split, conv3_tiles(v));
    const float zero[4] = {0.f, 0.f, 0.f, 0.f};
    float acc[4][4] = {}, low[4][4] = {};
    int toff[4];  // halo offsets of the warp's taps
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int tap = min(warp + 8 * q, 26);
        toff[q] = (tap / 9 * kHY + tap / 3 % 3) * kHX + tap % 3;
    }
    for (int i = t0; i < t1; ++i) {
        const Tile3 tl(i, v);
        if (tid < kPairs) {
            const int o0 = halo_offset(tid, tl, v), o1 = halo_offset(tid + kZPair, tl, v);
            float f[8][2];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float *x = a.x + (ci0 + c) * n;
                f[c][0] = ci0 + c < a.cin ? x[o0] : 0.f;
                f[c][1] = ci0 + c < a.cin ? x[o1] : 0.f;
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const Split3 sp(f[c][0], f[c][1]);
                xs[0][c][tid] = sp.h;
                xs[1][c][tid] = sp.m;
                xs[2][c][tid] = sp.l;
            }
        }
#pragma unroll
        for (int k = 0; k < kC3N * 64 / kThreads; ++k) {
            const int e = tid + kThreads * k, r = e & 63, c = e >> 6;
            const int x = tl.x0 + (r & 7), y = tl.y0 + (r >> 3 & 3), z = tl.z0 + (r >> 5);
            const bool on = x < v.w && y < v.h && co0 + c < a.cout;
            const float *d = a.dy + (co0 + c) * n + ((long long)z * v.h + y) * v.w + x;
            const Split3 sp(on && z < v.d ? d[0] : 0.f, on && z + 2 < v.d ? d[2LL * v.h * v.w] : 0.f);
            ds[0][c][r] = sp.h;
            ds[1][c][r] = sp.m;
            ds[2][c][r] = sp.l;
        }
        __syncthreads();
#pragma unroll 2
        for (int row = 0; row < 8; ++row) {  // eight voxels along x at (y, z) and at (y, z + 2)
            const int r = 8 * row + t, o = (row / 4 * kHY + row % 4) * kHX + t;
            uint32_t f[3][4];
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int j = 0; j < 4; ++j) f[k][j] = ds[k][g + 8 * (j & 1)][r + 4 * (j >> 1)];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int p = o + toff[q];
                uint32_t b[3][2];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    b[k][0] = xs[k][g][p];
                    b[k][1] = xs[k][g][p + 4];
                }
                float s[4], u[4];
                mma_bf16(u, f[0], b[0][0], b[0][1], zero);
                mma_bf16(s, f[2], b[0][0], b[0][1], zero);
                mma_bf16(s, f[0], b[2][0], b[2][1], s);
                mma_bf16(s, f[1], b[1][0], b[1][1], s);
                mma_bf16(s, f[1], b[0][0], b[0][1], s);
                mma_bf16(s, f[0], b[1][0], b[1][1], s);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    acc[q][k] += u[k];
                    low[q][k] += s[k];
                }
            }
        }
        __syncthreads();
    }
    float *dst = a.part + (long long)blockIdx.z * a.cout * a.cin * 27;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int tap = warp + 8 * q;
        if (tap > 26) break;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int co = co0 + g + 8 * (k >> 1), ci = ci0 + 2 * t + (k & 1);
            if (co < a.cout && ci < a.cin) dst[((long long)co * a.cin + ci) * 27 + tap] = acc[q][k] + low[q][k];
        }
    }
}

// a = GELU(z) (erf form)
__global__ void k_gelu(const float *__restrict__ z, float *__restrict__ out, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = gelu_f(z[i]);
}

// g *= GELU'(z)
__global__ void k_gelu_bwd(const float *__restrict__ z, float *__restrict__ g, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        g[i] *= gelu_grad(z[i]);
}

// y += x
__global__ void k_add(float *__restrict__ y, const float *__restrict__ x, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] += x[i];
}

// db[c] (+)= sum_v g[c][v]; a cluster of eight blocks per channel, FP64 partials in a fixed order
// (4 to 64 channels leave most of the chip idle with one block each: 16 channels at 48^3 16 us, now 10)
constexpr int kBiasBlocks = 8;
__global__ void __cluster_dims__(kBiasBlocks, 1, 1) __launch_bounds__(256) k_bias_grad(const float *__restrict__ g, float *__restrict__ db, long long nv, int accumulate) {
    __shared__ double red[256];
    const int c = blockIdx.x / kBiasBlocks, rank = blockIdx.x % kBiasBlocks;
    const float *p = g + (long long)c * nv;
    double s = 0.0;
    for (long long i = rank * 256 + threadIdx.x; i < nv; i += 4 * 256 * kBiasBlocks) {  // four loads in flight
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = i + k * 256 * kBiasBlocks < nv ? p[i + k * 256 * kBiasBlocks] : 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) s += v[k];
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    auto cl = cooperative_groups::this_cluster();
    cl.sync();
    if (rank == 0 && threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < kBiasBlocks; ++k) t += *cl.map_shared_rank(red, k);
        db[c] = accumulate ? db[c] + (float)t : (float)t;
    }
    cl.sync();
}

// masked squared error over C channels: loss = sum_v m_v sum_c (y - t)^2 * inv_norm,
// g = dloss/dy; per-block FP64 partials to part[blockIdx.x]
__global__ void __launch_bounds__(256) k_mse(const float *__restrict__ y, const float *__restrict__ t, const float *__restrict__ mask,
                                             float *__restrict__ g, double *__restrict__ part, int C, long long nv, float inv_norm) {
    __shared__ double red[256];
    double s = 0.0;
    for (long long v = blockIdx.x * 256LL + threadIdx.x; v < nv; v += (long long)gridDim.x * 256) {
        const float m = mask ? mask[v] : 1.f;
        for (int c = 0; c < C; ++c) {
            const float d = y[(long long)c * nv + v] - t[(long long)c * nv + v];
            g[(long long)c * nv + v] = 2.f * m * d * inv_norm;
            s += (double)(m * d * d);
        }
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0] * (double)inv_norm;
}

// acc[0] += sum of the first n partials (one thread block)
__global__ void k_sum_into(const double *__restrict__ part, int n, double *__restrict__ acc) {
    __shared__ double red[256];
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += 256) s += part[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) acc[0] += red[0];
}

// Adam (Kingma & Ba 2015) on the FP32 master parameters; the BF16 copy used by the
// kernels is rewritten.  gscale multiplies the accumulated gradient (1/batch).
__global__ void k_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       __nv_bfloat16 *__restrict__ pb, long long n, float lr, float b1, float b2, float eps, float c1, float c2,
                       float gscale) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i] * gscale;
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
        p[i] = pi;
        pb[i] = __float2bfloat16_rn(pi);
    }
}

__global__ void k_to_bf16(const float *__restrict__ p, __nv_bfloat16 *__restrict__ pb, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        pb[i] = __float2bfloat16_rn(p[i]);
}

}  // namespace wn
}  // namespace mdft
