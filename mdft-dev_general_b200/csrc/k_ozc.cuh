// Rotated OZ step (S3-S5 of src/module_energy_cproj_mrso.f90:441-674) of a C2v solvent (mrso 2),
// templated on the working precision T and the angular order MM.
//
// What is shared sets the split.  The points (+-ix, +-iy, iz) have one |q| and one polar angle,
// so the interpolated c(|q|) and the real rotation matrices D(beta) of R(q) = e^{-i mu' alpha} D
// (the recursion of src/module_rotation.f90:119-247 pairs indices as m = x + u in
// every term, so the phases factor out of it and D follows it in real arithmetic) belong to a cell
// (|ix|, |iy|, iz) of up to four (q, -q) pairs.  A CTA takes four consecutive cells = 16 pairs at a time; lane = side (q / -q) x 4 sign choices x 4
// cells, so every lane works on one point.  D and the azimuth phases of a cell depend on the
// grid alone and come from a table laid out at creation; c is interpolated once per cell into
// shared memory; both are read as broadcasts.  The projections of the 32 points sit in shared
// memory as [ip][lane] (no bank conflicts; neighbouring cells are neighbouring x: coalesced).
// The warps of the CTA share the work by (m, mu2) blocks in the two rotations and by chi blocks
// in the OZ sums, each block with its inputs or sums in registers and its loops unrolled.  A
// rotation block and a chi block read and write only their own entries, so everything is in
// place.
//
// Bound: shared-memory load bandwidth (76 % of the LSU's at FP64 mmax 3: every multiply-add of
// the OZ sums brings half a c value per lane from shared memory), FP64 pipe 27 %.  Against the
// warp-per-pair k_oz2 (its tables interpreted per pair, R(q) and c formed per pair):
//   FP64 64^3 mmax 3: 667 -> 110 us; 96^3 mmax 1: 1014 -> 47 us; 32^3 mmax 5: 1008 -> 102 us
//   FP32 64^3 mmax 5: 3841 -> 330 us; mmax 3, against a thread per pair: 101 -> 68 us
// at 235, 159, 92, 369 and 117 MB of plane traffic.
#pragma once

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "k_angular.cuh"
#include "k_fft.cuh"
#include "k_oz2.cuh"

namespace mdft {

constexpr int kOzcCells = 4;  // cells per step of a CTA
constexpr int kOzcLd = 5;     // padded cell row of the staged c: conflict-free writes along k
constexpr int kOzcMaxWarps = 8;
constexpr int kOzcMaxTasks = 6;  // rotation or chi blocks of one warp

// mrso 2: projections of m, first projection of m, columns and rows of a chi block
__host__ __device__ constexpr int ozc_nm(int m) { return m / 2 + 1; }
__host__ __device__ constexpr int ozc_poff(int m) {
    int s = 0;
    for (int k = 0; k < m; ++k) s += (2 * k + 1) * ozc_nm(k);
    return s;
}
__host__ __device__ constexpr int ozc_rows(int M, int chi) {
    int s = 0;
    for (int m = chi < 0 ? -chi : chi; m <= M; ++m) s += ozc_nm(m);
    return s;
}
__host__ __device__ constexpr int ozc_cols(int M, int chi) {
    int s = 0;
    for (int m = chi < 0 ? -chi : chi; m <= M; ++m) s += 2 * (m / 2) + 1;
    return s;
}
// first coefficient of chi block chi (chi = M + 1: their number)
__host__ __device__ constexpr int ozc_coff(int M, int chi) {
    int s = 0;
    for (int x = -M; x < chi; ++x) s += ozc_rows(M, x) * ozc_cols(M, x);
    return s;
}

// D entries kept: (l, m, m1) with m1 >= 0; D(l, -m, -m1) = (-1)^(m+m1) D(l, m, m1)
__host__ __device__ constexpr int ozc_eoff(int l) {
    int s = 0;
    for (int k = 0; k < l; ++k) s += (2 * k + 1) * (k + 1);
    return s;
}
__host__ __device__ constexpr int ozc_eidx(int l, int m, int m1) { return ozc_eoff(l) + (m + l) * (l + 1) + m1; }

// A cell's record, values of T: {table row of |q|, its weight, Re and Im of e^{-i k alpha} for
// qx, qy >= 0 (k = 1..M), D (levels 1..M)}
__host__ __device__ constexpr int ozc_rec_d(int M) { return 2 + 2 * M - 1; }  // D entry e at ozc_rec_d + e
__host__ __device__ constexpr int ozc_rec(int M) { return ozc_rec_d(M) + ozc_eoff(M + 1); }

// Blocks dealt to warps at compile time, longest first to the least loaded: (m << 4 | mu2) of
// the rotations and chi + M of the OZ sums.
__host__ __device__ constexpr int ozc_warps(int M) { return M == 0 ? 1 : M == 1 ? 2 : M <= 3 ? 4 : 8; }
template <int M> struct OzcTasks {
    unsigned char nrot[kOzcMaxWarps] = {}, rot[kOzcMaxWarps][kOzcMaxTasks] = {};
    unsigned char nchi[kOzcMaxWarps] = {}, chi[kOzcMaxWarps][kOzcMaxTasks] = {};
    __host__ __device__ constexpr OzcTasks() {
        int load[kOzcMaxWarps] = {};
        for (int m = M; m >= 0; --m)
            for (int mu2 = 0; mu2 < ozc_nm(m); ++mu2) {
                int w = 0;
                for (int v = 1; v < ozc_warps(M); ++v)
                    if (load[v] < load[w]) w = v;
                rot[w][nrot[w]++] = (unsigned char)(m << 4 | mu2);
                load[w] += (2 * m + 1) * (2 * m + 1);
            }
        for (int v = 0; v < kOzcMaxWarps; ++v) load[v] = 0;
        for (int i = 0; i <= 2 * M; ++i) {  // 0, 1, -1, 2, -2, ...: falling size
            const int x = (i & 1) ? (i + 1) / 2 : -(i / 2);
            int w = 0;
            for (int v = 1; v < ozc_warps(M); ++v)
                if (load[v] < load[w]) w = v;
            chi[w][nchi[w]++] = (unsigned char)(x + M);
            load[w] += ozc_rows(M, x) * ozc_cols(M, x);
        }
    }
};
template <int M> __constant__ constexpr OzcTasks<M> kOzcTasks{};

struct OzcArgs {
    int nx, ny, nz, hx, hy;  // h = n/2 + 1
    long long N;
    int ncell;
    int quirks;  // FP64: the reference's single-precision flushes of R and gamma
};

struct OzcSetup {
    int hx, hy, ncell, mmax;
    int quirks;
    double dq, twopi_lx, twopi_ly, twopi_lz;
};

// Recursion of src/module_rotation.f90:119-247 for D: per entry of levels 2.. three products
// c_t D[x_t] D[u_t] of a level-1 and a level l-1 entry (x | u << 16), D(l, m > 0, 0) through its
// mirror image.
inline void build_ozc_recipes(int M, std::vector<int> &xu, std::vector<double> &cf) {
    RotCoef rc;
    build_rot_coef(rc);
    for (int l = 2; l <= M; ++l)
        for (int mm = -l; mm <= l; ++mm)
            for (int m1 = 0; m1 <= l; ++m1) {
                const int m = (mm > 0 && m1 == 0) ? -mm : mm;
                const double sg = m != mm ? (double)neg1pow(mm) : 1.0;
                const int x1 = m1 < l ? 0 : 1, u1 = m1 < l ? m1 : m1 - 1;
                double c[3] = {0, 0, 0};
                if (m1 < l) {
                    if (m > -l && m < l) c[0] = rc.a[l][m + kRMax][m1 + kRMax];
                    if (m > -l) c[1] = rc.b[l][m + kRMax][m1 + kRMax];
                    if (m < l) c[2] = rc.b[l][-m + kRMax][m1 + kRMax];
                } else {
                    if (m > -l && m < l) c[0] = rc.c[l][m + kRMax];
                    if (m > -l) c[1] = rc.d[l][m + kRMax];
                    if (m < l) c[2] = rc.d[l][-m + kRMax];
                }
                const int xm[3] = {0, 1, -1};
                for (int t = 0; t < 3; ++t) {
                    const int um = m - xm[t];
                    const bool in = std::abs(um) <= l - 1 && c[t] != 0.0;
                    xu.push_back(in ? ozc_eidx(1, xm[t], x1) | (ozc_eidx(l - 1, um, u1) << 16) : 0);
                    cf.push_back(in ? sg * c[t] : 0.0);
                }
            }
}

// c table [nq][ncoef] reordered as [nq][chi][column][row]
inline std::vector<double> build_ozc_table(const Grid &g, const CTable &ct) {
    std::vector<int> src;
    for (int chi = -g.mmax; chi <= g.mmax; ++chi) {
        int col = 0;
        for (int n = std::abs(chi); n <= g.mmax; ++n)
            for (int nu2 = -(n / g.mrso); nu2 <= n / g.mrso; ++nu2, ++col)
                for (int m = std::abs(chi); m <= g.mmax; ++m)
                    for (int mu2 = 0; mu2 <= m / g.mrso; ++mu2) src.push_back(ct.ia_start[g.pidx(m, chi, mu2)] + col);
    }
    std::vector<double> t((size_t)ct.nq * ct.ncoef * 2);
    for (int iq = 0; iq < ct.nq; ++iq) {
        const double *a = &ct.c[(size_t)iq * ct.ncoef * 2];
        double *b = &t[(size_t)iq * ct.ncoef * 2];
        for (int k = 0; k < ct.ncoef; ++k) {
            b[2 * k] = a[2 * src[k]];
            b[2 * k + 1] = a[2 * src[k] + 1];
        }
    }
    return t;
}

template <typename T> __host__ __device__ constexpr size_t ozc_smem_bytes(int M) {
    return sizeof(typename Cplx<T>::t) * ((size_t)ozc_poff(M + 1) * 32 + (size_t)ozc_coff(M, M + 1) * kOzcLd) +
           sizeof(T) * (size_t)ozc_rec(M) * kOzcCells;
}

// The cells' records, once per handle: a warp per cell, FP64 throughout, rounded to T at the
// end.  The reference flushes R = e^{-i mu' alpha} D by its parts (|Re| or |Im| < epsilon(1.) = 2^-23
// vanishes, the other part is rounded to single precision, :491-492).  With quirks the records do it
// through the factors: where a phase lies within epsilon of an axis every entry of its mu' loses one
// part, so the phase is put on the axis and the entries are rounded; a D below epsilon vanishes.
// That is not the whole rule: a part that is below epsilon as a product only (a D of a few epsilon,
// the phase off the axes) stays here, and the entry's other part unrounded.  Over the cells of a
// grid: no entry up to mmax 2; 64^3 mmax 3 216 of 2.98 million, mmax 5 4784 of 10.2 million; each part
// off by at most epsilon.  Measured against the whole rule, 32^3 mmax 5 and 32x48x24 mmax 4: F 2e-16
// and 1e-15 of itself, the excess gradient 9e-13 and 3e-12 of its largest value (bars 1e-10 and 1e-8).
// k_oz2 (mixtures, other solvents) flushes R itself.
template <typename T>
__global__ void __launch_bounds__(128) k_ozc_records(T *__restrict__ rec, const int *__restrict__ rxu, const double *__restrict__ rcf, OzcSetup a) {
    __shared__ double Ds[4][ozc_eoff(kMaxMmax + 1)];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, M = a.mmax;
    const int cell = blockIdx.x * 4 + warp;
    if (cell >= a.ncell) return;
    double *D = Ds[warp];
    T *r = rec + (size_t)cell * ozc_rec(M);
    const int ia = cell % a.hx, ib = (cell / a.hx) % a.hy, iz = cell / (a.hx * a.hy);
    const double qx = ia * a.twopi_lx, qy = ib * a.twopi_ly, qz = iz * a.twopi_lz;
    const double rho2 = qx * qx + qy * qy, rho = sqrt(rho2), nrm = sqrt(rho2 + qz * qz);
    const double ex = rho > 0.0 ? qx / rho : 1.0, ey = rho > 0.0 ? -qy / rho : 0.0;
    const double eff = nrm / a.dq + 1.0;  // :534-539
    double px = 1.0, py = 0.0;
    unsigned axis = 1u;
    for (int k = 1; k <= M; ++k) {
        const double x = px * ex - py * ey, y = px * ey + py * ex;
        px = x;
        py = y;
        double sx = px, sy = py;
        if (a.quirks && fabs(px) < kEpsSp) { sx = 0.0; sy = py > 0 ? 1.0 : -1.0; axis |= 1u << k; }
        else if (a.quirks && fabs(py) < kEpsSp) { sx = px > 0 ? 1.0 : -1.0; sy = 0.0; axis |= 1u << k; }
        if (lane == 0) {
            r[2 * k] = (T)sx;
            r[2 * k + 1] = (T)sy;
        }
    }
    if (lane == 0) {
        const double cb = nrm > 0.0 ? qz / nrm : 1.0, h = nrm > 0.0 ? rho / nrm * 0.70710678118654752440084436210484903928 : 0.0;
        r[0] = (T)((int)eff - 1);
        r[1] = (T)(eff - (int)eff);
        D[0] = 1.0;
        if (M >= 1) {
            D[ozc_eidx(1, -1, 0)] = h;
            D[ozc_eidx(1, -1, 1)] = 0.5 * (1.0 - cb);
            D[ozc_eidx(1, 0, 0)] = cb;
            D[ozc_eidx(1, 0, 1)] = h;
            D[ozc_eidx(1, 1, 0)] = -h;
            D[ozc_eidx(1, 1, 1)] = 0.5 * (1.0 + cb);
        }
    }
    __syncwarp();
    for (int l = 2; l <= M; ++l) {
        for (int f = lane; f < (2 * l + 1) * (l + 1); f += 32) {
            const int e = ozc_eoff(l) + f, o = 3 * (e - ozc_eoff(2));
            double v = 0.0;
            for (int t = 0; t < 3; ++t) v += rcf[o + t] * D[rxu[o + t] & 0xffff] * D[rxu[o + t] >> 16];
            D[e] = v;
        }
        __syncwarp();
    }
    for (int l = 1; l <= M; ++l)
        for (int f = lane; f < (2 * l + 1) * (l + 1); f += 32) {
            const int m = f / (l + 1) - l;
            double v = D[ozc_eoff(l) + f];
            if (a.quirks && fabs(v) < kEpsSp) v = 0.0;
            else if (a.quirks && (axis >> (m < 0 ? -m : m) & 1)) v = (double)__double2float_rn(v);
            r[ozc_rec_d(M) + ozc_eoff(l) + f] = (T)v;
        }
}

// asynchronous copy of one value to shared memory (zero when !ok)
template <int B>
__device__ __forceinline__ void ozc_copy(void *dst, const void *src, bool ok) {
    if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "n"(B), "r"(ok ? B : 0) : "memory");
}

// e^{-i k alpha} of this lane's point from the cell's (qx, qy >= 0): qx -> -qx takes p to
// (-1)^k conj p, qy -> -qy to conj p
template <typename T>
__device__ __forceinline__ typename Cplx<T>::t ozc_phase(const T *rec, int k, T sgx, T sgy) {
    typename Cplx<T>::t p;
    p.x = rec[2 * k * kOzcCells];
    p.y = rec[(2 * k + 1) * kOzcCells] * sgy;
    if (k & 1) p.x *= sgx;
    else p.y *= sgx;
    return p;
}

// The loops over chi, and over the columns of a chi block, stay rolled where the unrolled code
// of all blocks would not stay in the instruction cache.
template <int M> constexpr int kOzcUnroll = M >= 4 ? 1 : 16;

// Forward rotation (:505-523) of block (M, mu2), in place: with t = p(mup) e^{-i mup alpha},
// u(chi) = sum_mup t(mup) D(mup, chi), each D entry with chi >= 0 also serving (-mup, -chi).
// b: the block's first entry for this lane (mup values ozc_nm(M) entries apart); Dm: the
// cell's D of this level; the -q side stores u(chi) at -chi with the sign (-1)^M.
template <typename T, int M>
__device__ __forceinline__ void ozc_fwd(typename Cplx<T>::t *b, const T *Dm, const T *rec, T sgx, T sgy, bool side) {
    using C = typename Cplx<T>::t;
    constexpr int st = ozc_nm(M) * 32;
    C t[2 * M + 1];
#pragma unroll
    for (int i = 0; i <= 2 * M; ++i) t[i] = b[i * st];
#pragma unroll
    for (int k = 1; k <= M; ++k) {
        const C p = ozc_phase<T>(rec, k, sgx, sgy);
        t[M + k] = cmul(t[M + k], p);
        t[M - k] = cmul(t[M - k], cconj(p));
    }
    const T sg = (side && (M & 1)) ? (T)-1 : (T)1;
    const int dir = side ? -st : st;
    C *mid = b + M * st;
#pragma unroll kOzcUnroll<M>
    for (int x = 0; x <= M; ++x) {
        C u, v;
        u.x = u.y = v.x = v.y = (T)0;
#pragma unroll
        for (int i = 0; i <= 2 * M; ++i) {
            const T d = Dm[(i * (M + 1) + x) * kOzcCells], e = ((i + M) & 1) ? -d : d;
            u.x = fma(d, t[i].x, u.x);
            u.y = fma(d, t[i].y, u.y);
            v.x = fma(e, t[2 * M - i].x, v.x);  // times (-1)^chi; x = 0: u once more
            v.y = fma(e, t[2 * M - i].y, v.y);
        }
        const T sv = (x & 1) ? -sg : sg;
        u.x *= sg; u.y *= sg;
        v.x *= sv; v.y *= sv;
        if (x > 0) mid[-x * dir] = v;
        mid[x * dir] = u;
    }
}

// Back rotation (:611-641) of block (M, mu2) straight to the planes: g the block's first value
// at this lane's point; conj: the -q result of a self-conjugate Nyquist point.
template <typename T, int M>
__device__ __forceinline__ void ozc_bwd(const typename Cplx<T>::t *b, const T *Dm, const T *rec, T sgx, T sgy, bool side,
                                        typename Cplx<T>::t *g, long long N, bool store, bool conj) {
    using C = typename Cplx<T>::t;
    constexpr int st = ozc_nm(M) * 32;
    C v[2 * M + 1];
    const int dir = side ? -st : st;
    const C *mid = b + M * st;
    {
        const C h0 = mid[0];
#pragma unroll
        for (int i = 0; i <= 2 * M; ++i) {
            const T d = M == 0 ? (T)1 : Dm[i * (M + 1) * kOzcCells];
            v[i].x = d * h0.x;
            v[i].y = d * h0.y;
        }
    }
#pragma unroll kOzcUnroll<M>
    for (int k = 1; k <= M; ++k) {
        C h0 = mid[k * dir], h1 = mid[-k * dir];
        if (k & 1) { h1.x = -h1.x; h1.y = -h1.y; }
#pragma unroll
        for (int i = 0; i <= 2 * M; ++i) {
            const T d = Dm[(i * (M + 1) + k) * kOzcCells], e = ((i + M) & 1) ? -d : d;
            v[i].x = fma(d, h0.x, v[i].x);
            v[i].y = fma(d, h0.y, v[i].y);
            v[2 * M - i].x = fma(e, h1.x, v[2 * M - i].x);
            v[2 * M - i].y = fma(e, h1.y, v[2 * M - i].y);
        }
    }
#pragma unroll
    for (int k = 1; k <= M; ++k) {
        const C p = ozc_phase<T>(rec, k, sgx, sgy);
        v[M + k] = cmul(v[M + k], cconj(p));
        v[M - k] = cmul(v[M - k], p);
    }
    if (!store) return;
    const T sg = (side && (M & 1)) ? (T)-1 : (T)1, sy = conj ? -sg : sg;
#pragma unroll
    for (int i = 0; i <= 2 * M; ++i) {
        C o;
        o.x = sg * v[i].x;
        o.y = sy * v[i].y;
        *g = o;
        g += ozc_nm(M) * N;
    }
}

// gamma flush of src/module_energy_cproj_mrso.f90:618-623
__device__ __forceinline__ double2 ozc_flush(double2 v) {
    if (fabs(v.x) < kEpsDp && fabs(v.y) < kEpsDp) return make_double2(0.0, 0.0);
    if (fabs(v.x) < kEpsDp) return make_double2(0.0, (double)__double2float_rn(v.y));
    if (fabs(v.y) < kEpsDp) return make_double2((double)__double2float_rn(v.x), 0.0);
    return v;
}
__device__ __forceinline__ float2 ozc_flush(float2 v) { return v; }

// OZ sums (:561-606) of chi block chi, |chi| = A: gamma(row) = sum_col c(row, col) x(col), x the
// lane's own r(n, chi, |nu2|) for nu2 < 0, the conjugate of the other side's otherwise.
template <typename T, int MM, int A>
__device__ __forceinline__ void ozc_chi(typename Cplx<T>::t *buf, const typename Cplx<T>::t *cc, int chi, int lane, int quirks) {
    using C = typename Cplx<T>::t;
    constexpr int R = ozc_rows(MM, A);
    C s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) s[r].x = s[r].y = (T)0;
#pragma unroll kOzcUnroll<MM>
    for (int n = A; n <= MM; ++n) {
        const int K = n / 2;
        const C *own = buf + (ozc_poff(n) + n * (K + 1)) * 32 + chi * ((K + 1) * 32) + lane;
        const C *oth = buf + (ozc_poff(n) + n * (K + 1)) * 32 + chi * ((K + 1) * 32) + (lane ^ 16);
#pragma unroll kOzcUnroll<MM>
        for (int nu2 = -K; nu2 <= K; ++nu2) {
            C x = nu2 < 0 ? own[-nu2 * 32] : oth[nu2 * 32];
            if (nu2 >= 0) x.y = -x.y;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const C c = cc[r * kOzcLd];
                s[r].x = fma(c.x, x.x, s[r].x);
                s[r].y = fma(c.x, x.y, s[r].y);
                s[r].x = fma(-c.y, x.y, s[r].x);
                s[r].y = fma(c.y, x.x, s[r].y);
            }
            cc += R * kOzcLd;
        }
    }
    __syncwarp();  // every lane has read the block
    int r = 0;
#pragma unroll
    for (int m = A; m <= MM; ++m)
#pragma unroll
        for (int mu2 = 0; mu2 < ozc_nm(m); ++mu2, ++r)
            buf[(ozc_poff(m) + m * ozc_nm(m) + mu2) * 32 + chi * (ozc_nm(m) * 32) + lane] = quirks ? ozc_flush(s[r]) : s[r];
}

// f(the compile-time value of v) for v in [0, MAX]
template <int V> struct OzcInt { static constexpr int v = V; };
template <int MAX, typename F>
__device__ __forceinline__ void ozc_for(int v, F f) {
    if (v == MAX) f(OzcInt<MAX>{});
    else if constexpr (MAX > 0) ozc_for<MAX - 1>(v, f);
}

template <typename T, int MM>
__global__ void __launch_bounds__(32 * ozc_warps(MM), 16 / ozc_warps(MM)) k_ozc(typename Cplx<T>::t *__restrict__ planes, const typename Cplx<T>::t *__restrict__ ctab,
                                                                                const T *__restrict__ records, const OzcArgs a) {
    using C = typename Cplx<T>::t;
    constexpr int NT = 32 * ozc_warps(MM), NP = ozc_poff(MM + 1), NC = ozc_coff(MM, MM + 1), RS = ozc_rec(MM);
    extern __shared__ __align__(16) unsigned char ozc_smem[];
    C *buf = reinterpret_cast<C *>(ozc_smem);               // [NP][32]
    C *cs = buf + NP * 32;                                  // [NC][kOzcLd]
    T *rec = reinterpret_cast<T *>(cs + NC * kOzcLd);       // [RS][kOzcCells]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool side = lane >= 16;
    const int j = lane & 3;
    const bool mx = lane & 4, my = lane & 8;  // -|ix|, -|iy|
    const T sgx = mx ? (T)-1 : (T)1, sgy = my ? (T)-1 : (T)1;
    pdl_launch();
    pdl_wait();
    for (int c0 = blockIdx.x * kOzcCells; c0 < a.ncell; c0 += gridDim.x * kOzcCells) {
        // ---- this lane's point ----
        const int cell = min(c0 + j, a.ncell - 1);
        const int row = cell / a.hx, ia = cell - row * a.hx, iz = row / a.hy, ib = row - iz * a.hy;
        const int iam = ia ? a.nx - ia : 0, ibm = ib ? a.ny - ib : 0, izm = iz ? a.nz - iz : 0;
        const int ix = mx ? iam : ia, iy = my ? ibm : ib, ixm = mx ? ia : iam, iym = my ? ib : ibm;
        bool active = c0 + j < a.ncell && !(mx && iam == ia) && !(my && ibm == ib);  // one sign only at 0 and Nyquist
        if (izm == iz && iy * a.nx + ix > iym * a.nx + ixm) active = false;           // the partner is the q
        const bool selfconj = ix == ixm && iy == iym && iz == izm;
        const bool nyq = 2 * ix == a.nx || 2 * iy == a.ny || 2 * iz == a.nz;
        C *own = planes + (side ? ((long long)izm * a.ny + iym) * a.nx + ixm : ((long long)iz * a.ny + iy) * a.nx + ix);
        {
            const C *src = own + warp * a.N;
#pragma unroll 4
            for (int ip = warp; ip < NP; ip += NT / 32, src += (NT / 32) * a.N) ozc_copy<sizeof(C)>(buf + ip * 32 + lane, src, active);
        }
        // ---- the cells' records ----
        for (int f = tid; f < RS * kOzcCells; f += NT) {
            const int q = f & 3, e = f >> 2;
            ozc_copy<sizeof(T)>(rec + f, records + (size_t)min(c0 + q, a.ncell - 1) * RS + e, true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        // ---- interpolated c (:534-539), once per cell ----
        {
            const C *p[kOzcCells];
            T al[kOzcCells];
#pragma unroll
            for (int q = 0; q < kOzcCells; ++q) {
                const T *r = records + (size_t)min(c0 + q, a.ncell - 1) * RS;
                p[q] = ctab + (size_t)(int)r[0] * NC;
                al[q] = r[1];
            }
#pragma unroll 2
            for (int k = tid; k < NC; k += NT) {
                C A[kOzcCells], B[kOzcCells];
#pragma unroll
                for (int q = 0; q < kOzcCells; ++q) {
                    A[q] = p[q][k];
                    B[q] = p[q][NC + k];
                }
#pragma unroll
                for (int q = 0; q < kOzcCells; ++q) {
                    C v;
                    v.x = al[q] * B[q].x + ((T)1 - al[q]) * A[q].x;
                    v.y = al[q] * B[q].y + ((T)1 - al[q]) * A[q].y;
                    cs[k * kOzcLd + q] = v;
                }
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const T *rj = rec + j;
        // ---- forward rotations ----
        for (int i = 0; i < kOzcTasks<MM>.nrot[warp]; ++i) {
            const int m = kOzcTasks<MM>.rot[warp][i] >> 4, mu2 = kOzcTasks<MM>.rot[warp][i] & 15;
            ozc_for<MM>(m, [&](auto mc) {
                constexpr int mm = decltype(mc)::v;
                if constexpr (mm > 0)  // mm 0: D = 1
                    ozc_fwd<T, mm>(buf + (ozc_poff(mm) + mu2) * 32 + lane, rj + (ozc_rec_d(MM) + ozc_eoff(mm)) * kOzcCells, rj, sgx, sgy, side);
            });
        }
        __syncthreads();
        // ---- OZ sums ----
        for (int i = 0; i < kOzcTasks<MM>.nchi[warp]; ++i) {
            const int chi = (int)kOzcTasks<MM>.chi[warp][i] - MM;
            ozc_for<MM>(chi < 0 ? -chi : chi, [&](auto xc) {
                constexpr int A = decltype(xc)::v;
                ozc_chi<T, MM, A>(buf, cs + (chi < 0 ? ozc_coff(MM, -A) : ozc_coff(MM, A)) * kOzcLd + j, chi, lane, a.quirks);
            });
        }
        __syncthreads();
        // ---- back rotations ----
        const bool store = active && !(selfconj && !side);  // self-conjugate points keep the -q result
        const bool cj = selfconj && nyq && side;
        for (int i = 0; i < kOzcTasks<MM>.nrot[warp]; ++i) {
            const int m = kOzcTasks<MM>.rot[warp][i] >> 4, mu2 = kOzcTasks<MM>.rot[warp][i] & 15;
            ozc_for<MM>(m, [&](auto mc) {
                constexpr int mm = decltype(mc)::v;
                ozc_bwd<T, mm>(buf + (ozc_poff(mm) + mu2) * 32 + lane, rj + (ozc_rec_d(MM) + ozc_eoff(mm)) * kOzcCells, rj, sgx, sgy, side,
                               own + (long long)(ozc_poff(mm) + mu2) * a.N, a.N, store, cj);
            });
        }
        __syncthreads();  // buf, c and the records are free
    }
}

}  // namespace mdft
