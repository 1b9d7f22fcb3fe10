// Angular transforms on the warp-level matrix instructions: S1 projection and S7 gather with the
// ideal and external terms (same arithmetic as the reference's, see k_angular.cuh), for every
// angular order and point count.  T = double: mma.sync m16n8k8 f64 (tcgen05 has no FP64 kind).
// T = float (FP32 planes, FP64 fields: FP32 evaluations of an FP64 point): m16n8k8 tf32 with both
// operands split in two, hi hi + hi lo + lo hi, FP32 accumulation.
//
// Both transforms are [points x K] . [K x J] products.  Why the matrix instructions: a DFMA reads
// three 8-byte registers per lane and reached 26 TFLOP/s here from registers alone, the matrix
// form 36.8 TFLOP/s with eight warps per SM, and it needs an eighth of the shared-memory loads;
// the FP32 form has 270 TFLOP/s, 90 after the split, against 71 of FFMA.
//
// Stage times (us) of evaluations back to back, project / gather, against the tiled FFMA and
// bulk-copy FFMA kernels before:
//   FP64 64^3 mmax 3: 189 -> 123 / 409 -> 228    FP64 96^3 mmax 1: 79 -> 20 / 400 -> 51
//   FP64 32^3 mmax 5: 1091 -> 189 / 1171 -> 285  FP32 64^3 mmax 5: 2740 -> 1240 / 3080 -> 1710
//   FP32 64^3 mmax 3: 104 / 202, where the tcgen05 forms for an FP64 point took 87 / 308 with ten
//   times the error (2.5e-6 of df against 2.1e-7, their BF16 halves): the projection alone is
//   slower here, the gather and the accuracy decide
// The matrix pipe is the floor (81 and 79 us at 64^3 mmax 3, padding of 8 included; 116 at 32^3
// mmax 5); the projection has it 66 % busy, the gather 35 % next to 43 us of epilogue on the
// FP64 pipe, its warps (16 per SM at 128 registers) waiting on loads, table reads and each other.
//
// A CTA keeps a chunk of the matrix (all of it up to mmax 3) in shared memory and walks tiles of
// BM points.  Their inputs come in K slabs through a ring of stages by bulk copies (a xi row that
// starts 8 bytes off a 16-byte boundary is copied from the value before it; xi itself off one
// goes by cp.async); eight warps, WM
// along the points (16 each) x WN along the columns (NT tiles of 8 each).  The order of K inside a
// block of 8 is free as long as both operands share it, so a lane takes two neighbouring K
// values by one load: re and im of a projection in the gather, two orientations in the
// projection.  The row strides keep these loads free of bank conflicts.
#pragma once

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "k_angular.cuh"
#include "k_tma.cuh"

namespace mdft {

constexpr int kDmWarps = 8;                          // compute warps of a CTA
constexpr int kPmThreads = 32 * (kDmWarps + 1);      // the projection has a copy warp
constexpr int kGmThreads = 32 * kDmWarps;
constexpr int kDmMaxStages = 4;

struct DmShape {
    int nkb = 0;     // K blocks of 8
    int skb = 0;     // K blocks per slab
    int nslab = 0;
    int nstage = 0;
    int ntc = 0;     // column tiles of 8 per chunk
    int nchunk = 0;
    int wn = 0, nt = 0;  // warps along the columns, column tiles per warp
    int nb = 0, sa = 0;  // row strides: the matrix in 16-byte units, a slab in its pairs
    int pitch = 0;       // projection: from one stage to the next, in the same pairs (gather: 4 skb slab rows)
    int bm = 0;
    size_t smem = 0;
    int grid = 0;
};

// One block of 8 of K for 16 rows x 8 columns: rows g, g + 8 and K pairs t of A, K pairs t and
// column g of B (16 bytes: the pair, or its hi and lo parts)
template <typename T> struct DmFrag;
template <> struct DmFrag<double> {
    double2 a0, a1;
    __device__ __forceinline__ DmFrag(double2 x0, double2 x1) : a0(x0), a1(x1) {}
    __device__ __forceinline__ void mma(double (&c)[4], double2 b) const {
        asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                     : "d"(a0.x), "d"(a1.x), "d"(a0.y), "d"(a1.y), "d"(b.x), "d"(b.y));
    }
};
__host__ __device__ inline float dm_tf32(float x) {  // to 11 significant bits, ties away
#ifdef __CUDA_ARCH__
    uint32_t u;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(x));
    return __uint_as_float(u);
#else
    uint32_t u;
    std::memcpy(&u, &x, 4);
    u = (u + 0x1000u) & 0xFFFFE000u;
    std::memcpy(&x, &u, 4);
    return x;
#endif
}
template <> struct DmFrag<float> {
    float hi[4], lo[4];
    __device__ __forceinline__ DmFrag(float2 x0, float2 x1) {
        const float v[4] = {x0.x, x1.x, x0.y, x1.y};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            hi[i] = dm_tf32(v[i]);
            lo[i] = dm_tf32(v[i] - hi[i]);
        }
    }
    static __device__ __forceinline__ void one(float (&c)[4], const float (&a)[4], double bxy) {
        asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
                       "r"(__double2loint(bxy)), "r"(__double2hiint(bxy)));
    }
    // The three products start from zero and are added to c in FP32: the tensor core's own
    // accumulation truncates, and a chain over all of K was 7.8e-6 off where this is 4e-7.
    __device__ __forceinline__ void mma(float (&c)[4], double2 b) const {
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        one(s, lo, b.x);
        one(s, hi, b.y);
        one(s, hi, b.x);
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] += s[i];
    }
};
__device__ __forceinline__ void dm_copy8(double *dst, const double *src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(ok ? 8 : 0) : "memory");
}
// an arrival on bar once this thread's cp.async so far have landed
__device__ __forceinline__ void dm_copy_arrive(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// The natural logarithm of a positive normal x, by the table method of Tang (ACM Trans. Math.
// Softw. 16 (1990) 378): x = 2^k m with m in [11/16, 11/8); with c ~ 1/m of the interval's table
// entry (1 around m = 1), log x = k ln 2 - log c + log1p(m c - 1), the last by its series to
// r^7 (|r| < 2^-7).  About 20 instructions against the library function's 70 in an epilogue
// that is issue-bound.  Absolute error below 3/2 2^-52 max(1, |log x|): each of the two last
// additions rounds by at most 2^-53 |log x|, ln 2's own rounding adds 0.15 2^-52 |log x|, the
// table's 2^-55 and the series' end with r's rounding 2^-58.
constexpr int kLogN = 128;
inline void dm_log_table(double2 *t) {
    for (int i = 0; i < kLogN; ++i) {
        // intervals of the upper seven mantissa bits, from 11/16 on
        const int j = i + 48;  // mantissa index of 11/16 in [1/2, 1) is 48
        const double lo = j < 128 ? 0.5 + j / 256.0 : 1.0 + (j - 128) / 128.0;
        const double hi = j < 128 ? lo + 1.0 / 256.0 : lo + 1.0 / 128.0;
        const double c = (lo == 1.0 || hi == 1.0) ? 1.0 : 2.0 / (lo + hi);
        t[i].x = c;
        t[i].y = -std::log(c);
    }
}
// the upper and lower word of a double, and back
__host__ __device__ __forceinline__ void dm_words(double x, int &hi, int &lo) {
#ifdef __CUDA_ARCH__
    hi = __double2hiint(x);
    lo = __double2loint(x);
#else
    int w[2];
    std::memcpy(w, &x, 8);
    lo = w[0];
    hi = w[1];
#endif
}
__host__ __device__ __forceinline__ double dm_double(int hi, int lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double(hi, lo);
#else
    const int w[2] = {lo, hi};
    double x;
    std::memcpy(&x, w, 8);
    return x;
#endif
}
__host__ __device__ __forceinline__ double dm_log(double x, const double2 *tab) {
    int h, l;
    dm_words(x, h, l);
    const int d = h - 0x3FE60000;
    const int k = d >> 20;
    const double2 e = tab[(d >> 13) & (kLogN - 1)];
    const double m = dm_double(h - (int)((unsigned)k << 20), l);
    const double kd = dm_double(0x43300000, k ^ 0x80000000) - 4503601774854144.0;  // (double)k
    const double r = fma(m, e.x, -1.0);
    double p = fma(r, 1.0 / 7.0, -1.0 / 6.0);
    p = fma(p, r, 1.0 / 5.0);
    p = fma(p, r, -1.0 / 4.0);
    p = fma(p, r, 1.0 / 3.0);
    p = fma(p, r, -1.0 / 2.0);
    return fma(kd, 0.69314718055994530941723212145817656808, e.y) + fma(r * r, p, r);
}

// Slab, stage and chunk sizes for K = 8 nkb and J columns: as few column chunks as the shared
// memory takes next to two slabs (each chunk reads the inputs again), then the longest slabs, then
// as many stages as do not cost a resident CTA.  a_bytes(skb, bm): bytes of one slab.
template <typename F>
inline DmShape dm_shape(int nkb, int J, size_t dyn_max, int max_stages, F a_bytes) {
    DmShape s;
    s.nkb = nkb;
    const int ntot = (J + 7) / 8;
    for (int nchunk = 1; nchunk <= ntot; ++nchunk) {
        const int ntc = (ntot + nchunk - 1) / nchunk;
        // four column warps from 5 tiles on (short point tiles: two CTAs per SM, or long slabs
        // next to a large matrix), two from 3, else all along the points
        const int wn = ntc > 4 ? 4 : ntc > 2 ? 2 : 1, nt = (ntc + wn - 1) / wn;
        if (nt > 4) continue;
        const int bm = 16 * (kDmWarps / wn);
        for (int nslab = 1; nslab <= nkb; ++nslab) {
            const int skb = (nkb + nslab - 1) / nslab;
            if (nslab > 1 && skb < 4) break;
            const int nb = wn * nt * 8 + 2;
            auto bytes = [&](int st) { return 16 * ((size_t)nkb * 4 * nb + wn * nt * 4 + kLogN) + st * (size_t)a_bytes(skb, bm); };
            if (bytes(2) > dyn_max) continue;
            const int ctas = (int)std::min<size_t>(2, (dyn_max - 2048) / bytes(2));
            s.nstage = 2;
            while (s.nstage < max_stages && (int)std::min<size_t>(2, (dyn_max - 2048) / bytes(s.nstage + 1)) == ctas) ++s.nstage;
            s.skb = skb;
            s.nslab = (nkb + skb - 1) / skb;
            s.ntc = ntc;
            s.nchunk = nchunk;
            s.wn = wn;
            s.nt = nt;
            s.nb = nb;
            s.bm = bm;
            s.smem = std::max(bytes(s.nstage), kReduceBytes);
            return s;
        }
    }
    return s;  // nt == 0: does not fit
}
// pairs of a slab row: the gather's [4 skb projections][bm + pad] (2 mod 8 pairs of doubles, 4
// mod 16 pairs of floats), the projection's [bm][row of 8 skb doubles, one more for the rows of
// an odd number of orientations, 4 mod 8 pairs]
inline int dm_row_pairs(int skb, int odd) { return (skb * 4 + odd + 3) / 8 * 8 + 4; }
template <typename T> inline int dm_gather_row(int bm) { return bm + (sizeof(T) == 8 ? 2 : 4); }
template <typename T>
inline DmShape dm_gather_shape(int np, int no, size_t dyn_max) {
    // Two stages: the fields' loads live in what shared memory leaves to L1.  At 64^3 mmax 3
    // three stages (215 of 228 KB) took 272 us, two (154 KB) 228.
    DmShape s = dm_shape((np + 3) / 4, no, dyn_max, 2, [](int skb, int bm) { return 4 * skb * dm_gather_row<T>(bm) * 2 * sizeof(T); });
    s.sa = dm_gather_row<T>(s.bm);
    return s;
}
template <typename T>
inline DmShape dm_project_shape(int np, int no, size_t dyn_max) {
    DmShape s = dm_shape((no + 7) / 8, 2 * np, dyn_max, kDmMaxStages,
                         [&](int skb, int bm) { return (size_t)bm * dm_row_pairs(skb, no & 1) * 16; });
    // short rows stay unpadded, a tile is one copy (a copy per 48-byte row bound the kernel: 96^3
    // mmax 1 110 us against 20); the K values past a row's end are its neighbour's, times zero, and
    // those past a tile's last row a pad after the stage, which no copy writes (the next stage may
    // be in flight).  The shorter rows leave room for it.
    s.sa = (no % 2 == 0 && no <= 16) ? no / 2 : dm_row_pairs(s.skb, no & 1);
    s.pitch = s.bm * s.sa + std::max(0, 4 * s.skb - s.sa);
    return s;
}

// Values written per row and slab of nu pairs where xi is copied 8 bytes at a time: the K padding
// is zeroed too, but never past the row, where an unpadded one is followed by the next row, the
// next stage or the matrix.
__host__ __device__ inline int dm_any_values(int nu, int sa) { return 2 * (nu < sa ? nu : sa); }

// The matrix in the order the kernels keep it, [chunk][4 nkb K pairs][nb] units of 16 bytes: the
// pair (T = double) or its hi and lo parts (float); value(k, j) is the FP64 entry, 0 outside.
template <typename T, typename F>
inline std::vector<double2> dm_image(const DmShape &s, F value) {
    std::vector<double2> img((size_t)s.nchunk * s.nkb * 4 * s.nb, make_double2(0.0, 0.0));
    size_t o = 0;
    for (int c = 0; c < s.nchunk; ++c)
        for (int kp = 0; kp < 4 * s.nkb; ++kp)
            for (int j = 0; j < s.nb; ++j, ++o) {
                if (j >= 8 * s.ntc) continue;
                const double v0 = value(2 * kp, 8 * s.ntc * c + j), v1 = value(2 * kp + 1, 8 * s.ntc * c + j);
                if (sizeof(T) == 8) {
                    img[o] = make_double2(v0, v1);
                } else {
                    const float h0 = dm_tf32((float)v0), h1 = dm_tf32((float)v1);
                    const float f[4] = {h0, h1, dm_tf32((float)(v0 - h0)), dm_tf32((float)(v1 - h1))};
                    std::memcpy(&img[o], f, 16);
                }
            }
    return img;
}

struct DmWalk {
    int nkb, skb, nslab, nstage, ntc, nchunk, nb, sa, pitch;
    int ntiles;
    __host__ __device__ DmWalk(const DmShape &s, long long N)
        : nkb(s.nkb), skb(s.skb), nslab(s.nslab), nstage(s.nstage), ntc(s.ntc), nchunk(s.nchunk), nb(s.nb), sa(s.sa), pitch(s.pitch),
          ntiles((int)((N + s.bm - 1) / s.bm)) {}
};

// The ring: full[s] completes when stage s has landed (narrive arrivals: one with the copies'
// bytes, or one per copying lane), empty[s] when every compute warp has read it.
struct DmRing {
    uint64_t full[kDmMaxStages], empty[kDmMaxStages];
    int abort;
};
// The chunk's matrix, zeroed slabs (the padding of K is never copied over) and the barriers.
__device__ __forceinline__ void dm_stage(DmRing &rg, int narrive, double2 *Bs, const double2 *bsrc, int nbu, double2 *As, int nau) {
    if (threadIdx.x == 0) {
        for (int i = 0; i < kDmMaxStages; ++i) {
            mbar_init(&rg.full[i], narrive);
            mbar_init(&rg.empty[i], kDmWarps);
        }
        mbar_fence_init();
        rg.abort = 0;
    }
    for (int f = threadIdx.x; f < nbu; f += blockDim.x) Bs[f] = bsrc[f];
    for (int f = threadIdx.x; f < nau; f += blockDim.x) As[f] = make_double2(0.0, 0.0);
    fence_proxy_async_smem();
    __syncthreads();
}
// The copy warp: load(tile, slab, stage) for each step as its stage comes free.
template <typename F>
__device__ __forceinline__ void dm_produce(DmRing &rg, const DmWalk &s, int first, int stride, int nsteps, F load) {
    int tile = first, slab = 0, st = 0, ph = 0;
    for (int i = 0; i < nsteps; ++i) {
        if (i >= s.nstage && !mbar_wait(&rg.empty[st], (uint32_t)(ph ^ 1))) {
            rg.abort = 1;
            return;
        }
        load(tile, slab, st);
        if (++slab == s.nslab) {
            slab = 0;
            tile += stride;
        }
        if (++st == s.nstage) {
            st = 0;
            ph ^= 1;
        }
    }
}
// All warps, after their loops: false when a wait ran out.  The copies still in flight get a
// bounded wait (a stage's barrier is at most one phase behind its last copy).
__device__ __forceinline__ bool dm_finish(DmRing &rg, const DmWalk &s, int nsteps, int *err) {
    __syncthreads();
    if (!rg.abort) return true;
    if (threadIdx.x == 0) {
        atomicExch(err, 1);
        for (int i = 0; i < min(nsteps, s.nstage); ++i)
            for (uint32_t p = 0; p < 2; ++p)
                if (!mbar_try_wait(&rg.full[i], p)) (void)mbar_wait(&rg.full[i], p);
    }
    return false;
}

// S1: xi [N][no] -> planes [np][N].  Rows of xi: 16-byte aligned (kRowEven); aligned at every
// other point (kRowOdd, no odd: an odd point's row is copied from 8 bytes before its start, so
// that copies stay aligned, and read one value further on); else copied 8 bytes at a time.
enum DmRows { kRowEven, kRowOdd, kRowAny };
template <typename T, int WN, int NT, int ROWS>
__global__ void __launch_bounds__(kPmThreads, 2) k_project_mma(const double *__restrict__ xi, const double2 *__restrict__ img,
                                                               typename Cplx<T>::t *__restrict__ planes, int *__restrict__ err, AngularArgs a, DmWalk s) {
    using C = typename Cplx<T>::t;
    constexpr int BM = 16 * (kDmWarps / WN);
    extern __shared__ __align__(128) unsigned char dm_smem[];
    __shared__ DmRing rg;
    double2 *As = reinterpret_cast<double2 *>(dm_smem);  // [stage: pitch][BM][sa]
    double2 *Bs = As + s.nstage * s.pitch;               // [4 nkb][nb]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk = blockIdx.x % s.nchunk, first = blockIdx.x / s.nchunk, stride = gridDim.x / s.nchunk;
    const int nsteps = first < s.ntiles ? ((s.ntiles - 1 - first) / stride + 1) * s.nslab : 0;
    pdl_launch();
    dm_stage(rg, ROWS != kRowAny ? 1 : 32, Bs, img + (size_t)chunk * s.nkb * 4 * s.nb, s.nkb * 4 * s.nb, As, s.nstage * s.pitch);
    pdl_wait();
    if (warp == kDmWarps) {
        dm_produce(rg, s, first, stride, nsteps, [&](int tile, int slab, int st) {
            const int u0 = slab * s.skb * 4, nu = min(s.skb, s.nkb - slab * s.skb) * 4;
            const int rows = (int)min((long long)BM, a.N - (long long)tile * BM);
            const double *src = xi + (long long)tile * BM * a.no + 2 * u0;
            if constexpr (ROWS == kRowOdd) {
                const int n = min(2 * nu, a.no - 2 * u0);  // rows even, odd: n, n + 1 values, in pairs
                const uint32_t b0 = 16u * (uint32_t)((n + 1) / 2), b1 = 16u * (uint32_t)((n + 2) / 2);
                if (lane == 0) mbar_arrive_expect_tx(&rg.full[st], (b0 + b1) * (rows / 2));
                __syncwarp();
                for (int r = lane; r < rows; r += 32)
                    bulk_load(As + st * s.pitch + r * s.sa, src + (long long)r * a.no - (r & 1), (r & 1) ? b1 : b0, &rg.full[st]);
            } else if constexpr (ROWS == kRowEven) {
                const uint32_t bytes = 16u * (uint32_t)min(nu, a.no / 2 - u0);
                if (lane == 0) mbar_arrive_expect_tx(&rg.full[st], bytes * rows);
                __syncwarp();
                if (2 * s.sa == a.no) {  // unpadded rows: one copy
                    if (lane == 0) bulk_load(As + st * s.pitch, src, bytes * rows, &rg.full[st]);
                } else {
                    for (int r = lane; r < rows; r += 32) bulk_load(As + st * s.pitch + r * s.sa, src + (long long)r * a.no, bytes, &rg.full[st]);
                }
            } else {
                const int n = dm_any_values(nu, s.sa);
                for (int r = 0; r < BM; ++r) {
                    double *dst = reinterpret_cast<double *>(As + st * s.pitch + r * s.sa);
                    for (int u = lane; u < n; u += 32) dm_copy8(dst + u, src + (long long)r * a.no + u, r < rows && 2 * u0 + u < a.no);
                }
                dm_copy_arrive(&rg.full[st]);
            }
        });
    } else {
        const int g = lane >> 2, t = lane & 3, wm = warp / WN, wn = warp % WN;
        T acc[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = (T)0;
        int tile = first, slab = 0, st = 0, ph = 0;
        for (int i = 0; i < nsteps; ++i) {
            if (!mbar_wait(&rg.full[st], (uint32_t)ph)) {
                rg.abort = 1;
                break;
            }
            const double2 *ar = As + st * s.pitch + (wm * 16 + g) * s.sa + t;
            const double2 *br = Bs + (slab * s.skb * 4 + t) * s.nb + wn * NT * 8 + g;
            const int nkb = min(s.skb, s.nkb - slab * s.skb);
#pragma unroll 2
            for (int kb = 0; kb < nkb; ++kb) {
                double2 x0, x1;
                if constexpr (ROWS == kRowOdd) {  // rows g, g + 8: of one parity
                    const double *r0 = reinterpret_cast<const double *>(ar + kb * 4) + (g & 1), *r1 = r0 + 16 * s.sa;
                    x0 = make_double2(r0[0], r0[1]);
                    x1 = make_double2(r1[0], r1[1]);
                } else {
                    x0 = ar[kb * 4];
                    x1 = ar[8 * s.sa + kb * 4];
                }
                C d0, d1;
                d0.x = (T)(a.rho0 * (x0.x * x0.x - 1.0));
                d0.y = (T)(a.rho0 * (x0.y * x0.y - 1.0));
                d1.x = (T)(a.rho0 * (x1.x * x1.x - 1.0));
                d1.y = (T)(a.rho0 * (x1.y * x1.y - 1.0));
                const DmFrag<T> f(d0, d1);
#pragma unroll
                for (int n = 0; n < NT; ++n) f.mma(acc[n], br[kb * 4 * s.nb + n * 8]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&rg.empty[st]);
            if (++st == s.nstage) {
                st = 0;
                ph ^= 1;
            }
            if (++slab == s.nslab) {  // the tile is complete: a column pair is one projection's (re, im)
                slab = 0;
                const long long p = (long long)tile * BM + wm * 16 + g;
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const int lt = wn * NT + n, ip = (chunk * s.ntc + lt) * 4 + t;
                    if (lt < s.ntc && ip < a.np) {
                        C *o = planes + (size_t)ip * a.N + p, v;
                        v.x = acc[n][0];
                        v.y = acc[n][1];
                        if (p < a.N) o[0] = v;
                        v.x = acc[n][2];
                        v.y = acc[n][3];
                        if (p + 8 < a.N) o[8] = v;
                    }
                    acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = (T)0;
                }
                tile += stride;
            }
        }
    }
    (void)dm_finish(rg, s, nsteps, err);
}

// two neighbouring values of a row (the second only where `two`); V16: one aligned access
template <typename TV, bool V16>
__device__ __forceinline__ double2 dm_load2(const TV *p, bool one, bool two) {
    if constexpr (V16 && sizeof(TV) == 8) {
        double2 v = make_double2(0.0, 0.0);
        if (one) v = *reinterpret_cast<const double2 *>(p);
        return v;
    } else {
        double2 v = make_double2(0.0, 0.0);
        if (one) v.x = (double)p[0];
        if (two) v.y = (double)p[1];
        return v;
    }
}

// S7 with the ideal + external term.  TD: type of df and of the search direction; V16: rows of
// xi, vext, df and d are 16-byte aligned (no even).  Column pairs of an accumulator are two
// neighbouring orientations, so a warp's accesses to the [N][no] fields are runs of 64 bytes.
template <typename T, int WN, int NT, bool V16, typename TD>
__global__ void __launch_bounds__(kGmThreads, NT <= 3 ? 2 : 1) k_gather_mma(const typename Cplx<T>::t *__restrict__ planes, const double2 *__restrict__ img,
                                                                            const double2 *__restrict__ logtab,
                                                                            const double *__restrict__ xi, const double *__restrict__ vext,
                                                                            const double *__restrict__ w, TD *__restrict__ df,
                                                                            double *__restrict__ partial, int *__restrict__ err, GatherArgs a, DmWalk s,
                                                                            SumsOut so) {
    using C = typename Cplx<T>::t;
    extern __shared__ __align__(128) unsigned char dm_smem[];
    pdl_launch();
    if (a.fail_wait) {  // the error path of a timed-out wait, with nothing issued yet
        pdl_wait();
        if (threadIdx.x == 0) atomicExch(err, 1);
        finish_gather(partial, so, reinterpret_cast<double *>(dm_smem));
        return;
    }
    constexpr int BM = 16 * (kDmWarps / WN), NC = WN * NT * 8;
    __shared__ DmRing rg;
    __shared__ double red[kGatherSums][kDmWarps];
    C *As = reinterpret_cast<C *>(dm_smem);                                   // [stage][4 skb][sa]
    double2 *Bs = reinterpret_cast<double2 *>(As + s.nstage * 4 * s.skb * s.sa);  // [4 nkb][nb]
    double2 *lt = Bs + s.nkb * 4 * s.nb;                                      // [kLogN]
    double *ws = reinterpret_cast<double *>(lt + kLogN);                      // [NC]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3, wm = warp / WN, wn = warp % WN;
    const int chunk = blockIdx.x % s.nchunk, first = blockIdx.x / s.nchunk, stride = gridDim.x / s.nchunk;
    const int col0 = chunk * s.ntc * 8, ncol = min(s.ntc * 8, a.no - col0);
    const int nsteps = first < s.ntiles ? ((s.ntiles - 1 - first) / stride + 1) * s.nslab : 0;
    const bool want_v = a.do_ideal != 0, want_d = a.df_mode == 1 && a.dvec != nullptr;
    const bool accum = a.df_mode == 2, store = a.df_mode != 0;  // accum: without the ideal term
    const double pre = a.prefactor * a.cst, x2min = kEpsDp / a.rho0, two_rho0 = 2.0 * a.rho0;
    for (int f = tid; f < NC; f += kGmThreads) ws[f] = f < ncol ? w[col0 + f] : 0.0;
    if (tid < kLogN) lt[tid] = logtab[tid];
    dm_stage(rg, 1, Bs, img + (size_t)chunk * s.nkb * 4 * s.nb, s.nkb * 4 * s.nb, reinterpret_cast<double2 *>(As),
             s.nstage * 4 * s.skb * s.sa * (int)sizeof(C) / 16);
    pdl_wait();
    int tl = first, sl = 0, stl = 0;  // the next slab to load and its stage
    auto load_next = [&]() {
        if (warp == 0) {  // a projection's points per copy
            const int ip0 = sl * s.skb * 4, nip = min(min(s.skb, s.nkb - sl * s.skb) * 4, a.np - ip0);
            const uint32_t bytes = (uint32_t)(min((long long)BM, a.N - (long long)tl * BM) * sizeof(C));
            if (lane == 0) mbar_arrive_expect_tx(&rg.full[stl], bytes * nip);
            __syncwarp();
            for (int ip = lane; ip < nip; ip += 32)
                bulk_load(As + (stl * 4 * s.skb + ip) * s.sa, planes + (size_t)(ip0 + ip) * a.N + (long long)tl * BM, bytes, &rg.full[stl]);
        }
        if (++sl == s.nslab) {
            sl = 0;
            tl += stride;
        }
        if (++stl == s.nstage) stl = 0;
    };
    for (int i = 0; i < s.nstage && i < nsteps; ++i) load_next();
    // sums over w-weighted elements; the constant factors go in at the end
    double fid = 0.0, fext = 0.0, fexc = 0.0, gdv = 0.0, gmx = 0.0, gun = 0.0;
    T acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = (T)0;
    const int cl = wn * NT * 8 + 2 * t;
    int tile = first, slab = 0, st = 0, ph = 0;
    for (int i = 0; i < nsteps; ++i) {
        const long long p0 = (long long)tile * BM + wm * 16 + g;
        const bool in0 = p0 < a.N, in1 = p0 + 8 < a.N, last = slab + 1 == s.nslab;
        const size_t e0 = (size_t)p0 * a.no + col0 + cl;
        // the tile's fields come in while its last slab is multiplied
        double2 xr[NT][2], vr[NT][2];
        if (last) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const double *xp = xi + e0 + (size_t)(8 * h) * a.no, *vp = vext + e0 + (size_t)(8 * h) * a.no;
                const bool in = h ? in1 : in0;
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const bool one = in && cl + 8 * n < ncol, two = in && cl + 8 * n + 1 < ncol;
                    xr[n][h] = dm_load2<double, V16>(xp + 8 * n, one, two);
                    vr[n][h] = dm_load2<double, V16>(vp + 8 * n, want_v && one, want_v && two);
                }
            }
        }
        if (!mbar_wait(&rg.full[st], (uint32_t)ph)) rg.abort = 1;
        const C *ar = As + (st * 4 * s.skb + t) * s.sa + wm * 16 + g;
        const double2 *br = Bs + (slab * s.skb * 4 + t) * s.nb + wn * NT * 8 + g;
        const int nkb = min(s.skb, s.nkb - slab * s.skb);
#pragma unroll 2
        for (int kb = 0; kb < nkb; ++kb) {
            const DmFrag<T> f(ar[kb * 4 * s.sa], ar[kb * 4 * s.sa + 8]);
#pragma unroll
            for (int n = 0; n < NT; ++n) f.mma(acc[n], br[kb * 4 * s.nb + n * 8]);
        }
        __syncthreads();  // the stage is free (and rg.abort visible)
        if (rg.abort) break;
        if (i + s.nstage < nsteps) load_next();
        if (++st == s.nstage) {
            st = 0;
            ph ^= 1;
        }
        if (!last) {
            ++slab;
            continue;
        }
        slab = 0;
        // no branch below, so that the elements of a thread interleave
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const double2 wr = *reinterpret_cast<const double2 *>(ws + cl + 8 * n);  // 0 past the chunk's columns
            const bool c0 = cl + 8 * n < ncol, c1 = cl + 8 * n + 1 < ncol;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const bool in = h ? in1 : in0, one = in && c0, two = in && c1;
                const size_t e = e0 + (size_t)(8 * h) * a.no + 8 * n;
                const double2 dv = dm_load2<TD, V16>(static_cast<const TD *>(a.dvec) + e, want_d && one, want_d && two);
                const double2 bv = dm_load2<TD, V16>(df + e, accum && one, accum && two);  // the excess gradient is added to it
                double2 gv;
                auto elem = [&](double x, double v, double d, double wio, double ac) {
                    const double x2 = x * x, wx2 = wio * x2;
                    const bool occ = want_v && x2 > x2min;  // rho > epsilon(1._dp)
                    const double l = dm_log(x2, lt), lg = occ ? l : 0.0, vo = occ ? v : 0.0;  // log(rho / rho0)
                    fexc = fma(wx2 - wio, ac, fexc);
                    fid = fma(wio, fma(x2, lg, 1.0 - x2), fid);
                    fext = fma(wx2, vo, fext);
                    const double gr = two_rho0 * wio * x * fma(pre, ac, fma(a.kT, lg, vo)), ga = fabs(gr);
                    gdv = fma(gr, d, gdv);
                    gmx = ga > gmx ? ga : gmx;
                    gun = fma(gr, wio, gun);
                    return gr;
                };
                gv.x = bv.x + elem(xr[n][h].x, vr[n][h].x, dv.x, in ? wr.x : 0.0, (double)acc[n][2 * h]);
                gv.y = bv.y + elem(xr[n][h].y, vr[n][h].y, dv.y, in ? wr.y : 0.0, (double)acc[n][2 * h + 1]);
                if constexpr (V16 && sizeof(TD) == 8) {
                    if (store && one) *reinterpret_cast<double2 *>(df + e) = gv;
                } else if constexpr (V16) {
                    if (store && one) *reinterpret_cast<float2 *>(df + e) = make_float2((float)gv.x, (float)gv.y);
                } else {
                    if (store && one) df[e] = (TD)gv.x;
                    if (store && two) df[e + 1] = (TD)gv.y;
                }
                acc[n][2 * h] = acc[n][2 * h + 1] = (T)0;
            }
        }
        tile += stride;
    }
    if (!dm_finish(rg, s, nsteps, err)) {
        finish_gather(partial, so, reinterpret_cast<double *>(dm_smem));
        return;
    }
    {
        for (int off = 16; off > 0; off >>= 1) {
            fid += __shfl_down_sync(0xffffffffu, fid, off);
            fext += __shfl_down_sync(0xffffffffu, fext, off);
            fexc += __shfl_down_sync(0xffffffffu, fexc, off);
            gdv += __shfl_down_sync(0xffffffffu, gdv, off);
            gmx = fmax(gmx, __shfl_down_sync(0xffffffffu, gmx, off));
            gun += __shfl_down_sync(0xffffffffu, gun, off);
        }
        if (lane == 0) {
            red[0][warp] = want_v ? fid * (a.kT * a.dv * a.rho0) : 0.0;
            red[1][warp] = fext * (a.dv * a.rho0);
            red[2][warp] = fexc * (pre * a.rho0);
            red[3][warp] = gdv;
            red[4][warp] = gmx;
            red[5][warp] = gun;
        }
    }
    __syncthreads();
    if (tid < kGatherSums) {
        double v = red[tid][0];
        for (int k = 1; k < kDmWarps; ++k) v = tid == 4 ? fmax(v, red[tid][k]) : v + red[tid][k];
        partial[kGatherSums * (size_t)blockIdx.x + tid] = v;
    }
    finish_gather(partial, so, reinterpret_cast<double *>(dm_smem));  // its stages are done
}

}  // namespace mdft
