// Batched 3-D FFTs over the projection planes, templated on precision and length.
//
// A length N = R1 R2 takes two register passes with one exchange through shared memory: with
// n = R2 a + b and k = k1 + R1 k2, a thread transforms the R1 values of one b, multiplies by
// w_N^(b k1), and after the exchange a thread transforms the R2 values of one k1.  The first
// pass reads global memory and the last one writes it, so a value crosses shared memory once
// per exchange and nothing is staged.
//
//  k_fft_xy<T, N>    a CTA per N x N plane: x, then y; three exchanges for both axes
//  k_fft_lines<T, N> the x axis alone (planes that are not square): a CTA per tile of lines
//  k_fft_cols<T, N>  the y or z axis: a CTA per tile of neighbouring columns
//
// Rows of shared memory hold Y[k1, b] at k1 P + b with P odd: lanes over b and lanes over k1
// both fall on distinct banks.  The second x pass leaves its outputs in its inputs' places (so
// no barrier separates them), the y passes pick column k1 + R1 k2 there, and the first y pass is
// in place too.  sign = +1: X[k] = sum_j x[j] e^{+2 pi i jk/N} (plan3dp of
// src/module_energy_cproj_mrso.f90:260); sign = -1: plan3dm; no scaling.
//
// Lengths: 8, 12, 16, 18, 24, 32, 36, 48, 54, 64, 72, 96 and 128; the others (below 8, 108, from 144
// on) run k_fft_axis.
#pragma once

#include "common.cuh"
#include "k_angular.cuh"
#include "k_fft.cuh"

namespace mdft {

__host__ __device__ constexpr int fft_r1(int n) {
    return n == 8 || n == 12 || n == 16 ? 4 : n == 18 || n == 24 || n == 36 ? 6 : n == 54 || n == 72 ? 9 : n == 96 ? 12 : n == 128 ? 16 : 8;
}
__host__ __device__ constexpr int fft_r2(int n) { return n / fft_r1(n); }
__host__ __device__ constexpr int fft_pitch(int n) { return fft_r2(n) | 1; }
__host__ __device__ constexpr int fft_row(int n) { return fft_r1(n) * fft_pitch(n); }

// w = e^{S 2 pi i / ...} times v for the constants of the small DFTs
template <int S, typename C> __device__ __forceinline__ C fft_muli(C v) {  // S i v
    C r;
    r.x = S > 0 ? -v.y : v.y;
    r.y = S > 0 ? v.x : -v.x;
    return r;
}
template <int S, typename C, typename T> __device__ __forceinline__ C fft_mulc(C v, T c, T s) {  // (c + S i s) v
    C r;
    const T t = S > 0 ? s : -s;
    r.x = c * v.x - t * v.y;
    r.y = c * v.y + t * v.x;
    return r;
}
template <typename T, int R, int S> struct Dft;
template <typename T, int S> struct Dft<T, 2, S> {
    using C = typename Cplx<T>::t;
    static __device__ __forceinline__ void run(C *v) {
        const C a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};
template <typename T, int S> struct Dft<T, 3, S> {
    using C = typename Cplx<T>::t;
    static __device__ __forceinline__ void run(C *v) {
        const T s3 = (T)(S * 0.86602540378443864676372317075293618);
        const C s = cadd(v[1], v[2]), d = csub(v[1], v[2]);
        C m, r;
        m.x = v[0].x - (T)0.5 * s.x;
        m.y = v[0].y - (T)0.5 * s.y;
        r.x = -s3 * d.y;
        r.y = s3 * d.x;
        v[0] = cadd(v[0], s);
        v[1] = cadd(m, r);
        v[2] = csub(m, r);
    }
};
template <typename T, int S> struct Dft<T, 4, S> {
    using C = typename Cplx<T>::t;
    static __device__ __forceinline__ void run(C *v) {
        const C a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = fft_muli<S>(csub(v[1], v[3]));
        v[0] = cadd(a, c);
        v[1] = cadd(b, d);
        v[2] = csub(a, c);
        v[3] = csub(b, d);
    }
};
template <typename T, int S> struct Dft<T, 8, S> {
    using C = typename Cplx<T>::t;
    static __device__ __forceinline__ void run(C *v) {
        const T h = (T)0.70710678118654752440084436210484903928;
        C a[4], b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            a[j] = cadd(v[j], v[j + 4]);
            b[j] = csub(v[j], v[j + 4]);
        }
        b[1] = fft_mulc<S>(b[1], h, h);
        b[2] = fft_muli<S>(b[2]);
        b[3] = fft_mulc<S>(b[3], -h, h);
        Dft<T, 4, S>::run(a);
        Dft<T, 4, S>::run(b);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[2 * k] = a[k];
            v[2 * k + 1] = b[k];
        }
    }
};
// coprime factors A B: n = (B n1 + A n2) mod AB, k = k1 mod A = k2 mod B, no twiddles
template <typename T, int A, int B, int S>
__device__ __forceinline__ void dft_coprime(typename Cplx<T>::t *v) {
    using C = typename Cplx<T>::t;
    C u[A][B];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1)
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) u[n1][n2] = v[(B * n1 + A * n2) % (A * B)];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) Dft<T, B, S>::run(u[n1]);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) {
        C w[A];
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) w[n1] = u[n1][k2];
        Dft<T, A, S>::run(w);
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) u[k1][k2] = w[k1];
    }
#pragma unroll
    for (int k = 0; k < A * B; ++k) v[k] = u[k % A][k % B];
}
template <typename T, int S> struct Dft<T, 6, S> {
    static __device__ __forceinline__ void run(typename Cplx<T>::t *v) { dft_coprime<T, 2, 3, S>(v); }
};
template <typename T, int S> struct Dft<T, 12, S> {
    static __device__ __forceinline__ void run(typename Cplx<T>::t *v) { dft_coprime<T, 3, 4, S>(v); }
};
// A A: n = A n1 + n2, k = k1 + A k2, twiddles w^(n2 k1) from the constants c, s
template <typename T, int A, int S>
__device__ __forceinline__ void dft_square(typename Cplx<T>::t *v, const T (&cs)[(A - 1) * (A - 1) + 1], const T (&sn)[(A - 1) * (A - 1) + 1]) {
    using C = typename Cplx<T>::t;
    C u[A][A];  // [n2][k1]
#pragma unroll
    for (int n2 = 0; n2 < A; ++n2) {
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) u[n2][n1] = v[A * n1 + n2];
        Dft<T, A, S>::run(u[n2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
        C w[A];
#pragma unroll
        for (int n2 = 0; n2 < A; ++n2) w[n2] = n2 * k1 == 0 ? u[n2][k1] : fft_mulc<S>(u[n2][k1], cs[n2 * k1], sn[n2 * k1]);
        Dft<T, A, S>::run(w);
#pragma unroll
        for (int k2 = 0; k2 < A; ++k2) v[k1 + A * k2] = w[k2];
    }
}
template <typename T, int S> struct Dft<T, 9, S> {
    static __device__ __forceinline__ void run(typename Cplx<T>::t *v) {
        const T c[5] = {(T)1, (T)0.76604444311897803520239265055541667, (T)0.17364817766693034885171662676931480, 0, (T)-0.93969262078590838405410927732473147};
        const T s[5] = {(T)0, (T)0.64278760968653932632264340990726343, (T)0.98480775301220805936674302458952302, 0, (T)0.34202014332566873304409961468225958};
        dft_square<T, 3, S>(v, c, s);
    }
};
template <typename T, int S> struct Dft<T, 16, S> {
    static __device__ __forceinline__ void run(typename Cplx<T>::t *v) {
        const T a = (T)0.92387953251128675612818318939678829, b = (T)0.38268343236508977172845998403039887, h = (T)0.70710678118654752440084436210484904;
        const T c[10] = {(T)1, a, h, b, (T)0, 0, -h, 0, 0, -a};
        const T s[10] = {(T)0, b, h, a, (T)1, 0, h, 0, 0, -b};
        dft_square<T, 4, S>(v, c, s);
    }
};

// Y[k1, b] = w_N^(b k1) DFT_R1 of v, w from the table of e^{+2 pi i t/N}
template <typename T, int N, int S>
__device__ __forceinline__ void fft_first(typename Cplx<T>::t *v, int b, const typename Cplx<T>::t *tw) {
    constexpr int R1 = fft_r1(N);
    Dft<T, R1, S>::run(v);
#pragma unroll
    for (int k = 1; k < R1; ++k) {
        typename Cplx<T>::t w = tw[b * k];  // b k < N
        if (S < 0) w.y = -w.y;
        v[k] = cmul(v[k], w);
    }
}

template <typename T, int N> __host__ __device__ constexpr int fft_xy_threads() { return N >= 72 ? 512 : N >= 32 ? 256 : 128; }
template <typename T, int N> __host__ __device__ constexpr size_t fft_xy_smem() { return sizeof(typename Cplx<T>::t) * ((size_t)N * fft_row(N) + N); }
template <typename T, int N> __host__ __device__ constexpr bool fft_xy_fits() { return fft_xy_smem<T, N>() <= 220 * 1024; }
// CTAs per SM the register allocator is asked to allow
template <typename T, int N> __host__ __device__ constexpr int fft_xy_blocks() {
    const int by_smem = (int)(220 * 1024 / fft_xy_smem<T, N>()), by_regs = 65536 / (fft_xy_threads<T, N>() * (sizeof(T) == 8 ? 80 : 48));
    const int b = by_smem < by_regs ? by_smem : by_regs;
    return b < 1 ? 1 : b;
}

template <typename T, int N, int S>
__global__ void __launch_bounds__(fft_xy_threads<T, N>(), fft_xy_blocks<T, N>()) k_fft_xy(typename Cplx<T>::t *__restrict__ data, const typename Cplx<T>::t *__restrict__ tw) {
    using C = typename Cplx<T>::t;
    constexpr int R1 = fft_r1(N), R2 = fft_r2(N), P = fft_pitch(N), ROW = fft_row(N), THREADS = fft_xy_threads<T, N>();
    extern __shared__ __align__(16) unsigned char fft_smem_[];
    C *twl = reinterpret_cast<C *>(fft_smem_), *buf = twl + N;
    C *g = data + (size_t)blockIdx.x * N * N;
    const int tid = threadIdx.x;
    pdl_launch();
    for (int i = tid; i < N; i += THREADS) twl[i] = tw[i];
    pdl_wait();
    // along x, R1: item (line, b)
    constexpr int I1 = N * R2, PER1 = (I1 + THREADS - 1) / THREADS;
    C v[R1];
#pragma unroll 1
    for (int q = 0; q < PER1; ++q) {
        const int it = tid + q * THREADS;
        const bool on = I1 % THREADS == 0 || it < I1;
        const int b = it % R2, line = it / R2;
        if (on) {
#pragma unroll
            for (int r = 0; r < R1; ++r) v[r] = g[line * N + r * R2 + b];
        }
        if (q == 0) __syncthreads();  // the table, with the first loads in flight
        if (on) {
            fft_first<T, N, S>(v, b, twl);
#pragma unroll
            for (int k = 0; k < R1; ++k) buf[line * ROW + k * P + b] = v[k];
        }
    }
    __syncthreads();
    // along x, R2: item (line, k1), in place
    constexpr int I2 = N * R1;
    for (int it = tid; it < I2; it += THREADS) {
        C u[R2];
        C *p = buf + (it / R1) * ROW + (it % R1) * P;
#pragma unroll
        for (int r = 0; r < R2; ++r) u[r] = p[r];
        Dft<T, R2, S>::run(u);
#pragma unroll
        for (int r = 0; r < R2; ++r) p[r] = u[r];
    }
    __syncthreads();
    // along y, R1: item (b, x), in place; column x = k1 + R1 k2 sits at k1 P + k2
    for (int it = tid; it < I1; it += THREADS) {
        const int x = it % N, b = it / N;
        C *p = buf + b * ROW + (x % R1) * P + x / R1;
#pragma unroll
        for (int r = 0; r < R1; ++r) v[r] = p[r * R2 * ROW];
        fft_first<T, N, S>(v, b, twl);
#pragma unroll
        for (int k = 0; k < R1; ++k) p[k * R2 * ROW] = v[k];
    }
    __syncthreads();
    // along y, R2: item (k1, x), to global memory
    for (int it = tid; it < I2; it += THREADS) {
        const int x = it % N, k1 = it / N;
        C u[R2];
        const C *p = buf + k1 * R2 * ROW + (x % R1) * P + x / R1;
#pragma unroll
        for (int r = 0; r < R2; ++r) u[r] = p[r * ROW];
        Dft<T, R2, S>::run(u);
#pragma unroll
        for (int r = 0; r < R2; ++r) g[(k1 + R1 * r) * N + x] = u[r];
    }
}

constexpr int kFftLines = 32, kFftLineThreads = 128;
template <typename T, int N> __host__ __device__ constexpr size_t fft_lines_smem() { return sizeof(typename Cplx<T>::t) * ((size_t)kFftLines * fft_row(N) + N); }

// lines of N contiguous values
template <typename T, int N, int S>
__global__ void __launch_bounds__(kFftLineThreads) k_fft_lines(typename Cplx<T>::t *__restrict__ data, const typename Cplx<T>::t *__restrict__ tw, long long nlines) {
    using C = typename Cplx<T>::t;
    constexpr int R1 = fft_r1(N), R2 = fft_r2(N), P = fft_pitch(N), ROW = fft_row(N);
    extern __shared__ __align__(16) unsigned char fft_smem_[];
    C *twl = reinterpret_cast<C *>(fft_smem_), *buf = twl + N;
    const long long l0 = (long long)blockIdx.x * kFftLines;
    const int lines = (int)min((long long)kFftLines, nlines - l0), tid = threadIdx.x;
    C *g = data + l0 * N;
    pdl_launch();
    for (int i = tid; i < N; i += kFftLineThreads) twl[i] = tw[i];
    __syncthreads();
    pdl_wait();
    for (int it = tid; it < lines * R2; it += kFftLineThreads) {
        const int b = it % R2, line = it / R2;
        C v[R1];
#pragma unroll
        for (int r = 0; r < R1; ++r) v[r] = g[line * N + r * R2 + b];
        fft_first<T, N, S>(v, b, twl);
#pragma unroll
        for (int k = 0; k < R1; ++k) buf[line * ROW + k * P + b] = v[k];
    }
    __syncthreads();
    for (int it = tid; it < lines * R1; it += kFftLineThreads) {
        const int k1 = it % R1, line = it / R1;
        C u[R2];
#pragma unroll
        for (int r = 0; r < R2; ++r) u[r] = buf[line * ROW + k1 * P + r];
        Dft<T, R2, S>::run(u);
#pragma unroll
        for (int r = 0; r < R2; ++r) g[line * N + k1 + R1 * r] = u[r];
    }
}

template <typename T> __host__ __device__ constexpr int fft_cols() { return sizeof(T) == 8 ? 16 : 32; }  // 256 bytes of a row
template <typename T, int N> __host__ __device__ constexpr int fft_col_threads() {
    const int items = fft_cols<T>() * (fft_r1(N) > fft_r2(N) ? fft_r1(N) : fft_r2(N));
    return items >= 256 ? 256 : 128;
}
template <typename T, int N> __host__ __device__ constexpr size_t fft_cols_smem() { return sizeof(typename Cplx<T>::t) * ((size_t)N * fft_cols<T>() + N); }

// columns c < ncol at (c / inner) outer + c % inner, N values es apart
template <typename T, int N, int S>
__global__ void __launch_bounds__(fft_col_threads<T, N>()) k_fft_cols(typename Cplx<T>::t *__restrict__ data, const typename Cplx<T>::t *__restrict__ tw,
                                                                      long long ncol, unsigned inner, long long outer, long long es) {
    using C = typename Cplx<T>::t;
    constexpr int R1 = fft_r1(N), R2 = fft_r2(N), TL = fft_cols<T>(), THREADS = fft_col_threads<T, N>();
    extern __shared__ __align__(16) unsigned char fft_smem_[];
    C *twl = reinterpret_cast<C *>(fft_smem_), *buf = twl + N;  // buf[slot][TL]
    const int tid = threadIdx.x, l = tid % TL;
    const long long c = (long long)blockIdx.x * TL + l;
    const bool on = c < ncol;
    C *g = data + (on ? (long long)(c / inner) * outer + c % inner : 0);
    pdl_launch();
    for (int i = tid; i < N; i += THREADS) twl[i] = tw[i];
    pdl_wait();
    constexpr int STEP = THREADS / TL;
#pragma unroll 1
    for (int q = 0; q < (R2 + STEP - 1) / STEP; ++q) {
        const int b = tid / TL + q * STEP;
        C v[R1];
        if (on && b < R2) {
#pragma unroll
            for (int r = 0; r < R1; ++r) v[r] = g[(r * R2 + b) * es];
        }
        if (q == 0) __syncthreads();  // the table, with the first loads in flight
        if (on && b < R2) {
            fft_first<T, N, S>(v, b, twl);
#pragma unroll
            for (int k = 0; k < R1; ++k) buf[(k * R2 + b) * TL + l] = v[k];
        }
    }
    __syncthreads();
    if (!on) return;
    for (int k1 = tid / TL; k1 < R1; k1 += STEP) {
        C u[R2];
#pragma unroll
        for (int r = 0; r < R2; ++r) u[r] = buf[(k1 * R2 + r) * TL + l];
        Dft<T, R2, S>::run(u);
#pragma unroll
        for (int r = 0; r < R2; ++r) g[(k1 + R1 * r) * es] = u[r];
    }
}

}  // namespace mdft
