// What the angular transforms share: their arguments and the reduction of the gathers' sums.
//
//  project (S1, src/module_energy_cproj_mrso.f90:276-290 with angl2proj):
//     drho_p[ip][r] = sum_io rho0 (xi[r][io]^2 - 1) A[io][ip]
//  gather (S7, src/module_energy_cproj_mrso.f90:728-762 with proj2angl), fused
//  with the ideal and external terms (src/module_energy_ideal_and_external.f90:46-73):
//     vexc[r][io] = P w(io) sum_ip gamma_p[ip][r]/N . B[ip][io]
//
// FP64 points: k_angular_mma.cuh; FP32 points and the resident tensor-core forms:
// k_angular_umma.cuh, k_project_tma.cuh, k_gather_tma.cuh.
#pragma once

#include "common.cuh"
#include "k_fft.cuh"

namespace mdft {

struct AngularArgs {
    long long N;  // points
    int no, np;
    double rho0;
};

// per-block partials of the gathers: F_id, F_ext, F_exc sum, df.d, max|df|, sum w df
constexpr int kGatherSums = 6;

struct GatherArgs {
    long long N;
    int no, np;
    double rho0, kT, dv, prefactor, cst;  // prefactor = -kT 2 (4 pi^2)/mrso/n0, cst = 1/N
    int do_ideal;                         // add F_id, F_ext and their gradient
    int df_mode;                          // 0 none, 1 store (id + exc), 2 accumulate exc
    const void *dvec;                     // df_mode 1: also df.dvec (null: df.df is not wanted -> 0);
                                          // FP64, or FP32 where df is
    int fail_wait;                        // the bulk-copy gathers report a timed-out wait at once,
                                          // before any copy or tensor-memory allocation (tests)
};

// Where an evaluation's sums go: the device copy (later kernels add to it) and, so that no copy
// follows the pipeline, pinned host memory together with the error flag.
struct SumsOut {
    double *sums, *host;
    const int *err;
    int *host_err;
    unsigned *count;  // CTAs of the running gather that are done
};

// One CTA of 256 threads: the n rows of kGatherSums partials into o, in a fixed order; entry 4 is
// a maximum, the others sums.  red: kGatherSums x 256 of shared memory.
constexpr size_t kReduceBytes = sizeof(double) * kGatherSums * 256;
__device__ __forceinline__ void reduce_rows(const double *partial, int n, const SumsOut &o, double *red) {
    const int t = threadIdx.x;
    double a[kGatherSums] = {0, 0, 0, 0, 0, 0};
    for (int i = t; i < n; i += 256)
#pragma unroll
        for (int j = 0; j < kGatherSums; ++j) {
            const double v = __ldcg(partial + (size_t)kGatherSums * i + j);
            a[j] = j == 4 ? fmax(a[j], v) : a[j] + v;
        }
#pragma unroll
    for (int j = 0; j < kGatherSums; ++j) red[256 * j + t] = a[j];
    __syncthreads();
    for (int off = 128; off > 0; off >>= 1) {
        if (t < off)
#pragma unroll
            for (int j = 0; j < kGatherSums; ++j) {
                double *r = red + 256 * j + t;
                *r = j == 4 ? fmax(r[0], r[off]) : r[0] + r[off];
            }
        __syncthreads();
    }
    if (t < kGatherSums) {
        o.sums[t] = red[256 * t];
        o.host[t] = red[256 * t];
    } else if (t == kGatherSums) {
        *o.host_err = *(const volatile int *)o.err;
    }
}

__global__ void __launch_bounds__(256) k_reduce_sums(const double *__restrict__ partial, int n, SumsOut o) {
    __shared__ double red[kGatherSums * 256];
    reduce_rows(partial, n, o, red);
}

// The last CTA (of 256 threads) of a gather to get here, its row of partials written or its
// failure flagged, reduces the rows: no launch of its own for it.  red: kReduceBytes.
__device__ __forceinline__ void finish_gather(const double *partial, const SumsOut &o, double *red) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(o.count, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    reduce_rows(partial, (int)gridDim.x, o, red);
    if (threadIdx.x == 0) *o.count = 0;
}

// sums[from ..] to the host copy, after kernels that follow the gather
__global__ void k_publish_sums(SumsOut o, int from, int to) {
    if ((int)threadIdx.x >= from && (int)threadIdx.x < to) o.host[threadIdx.x] = o.sums[threadIdx.x];
}

// Programmatic dependent launch: a kernel launched with it may begin while the one before it in
// the stream drains.  Everything that kernel wrote, or may still read, is touched only after
// pdl_wait; pdl_launch lets the next kernel's CTAs come as soon as there is room.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace mdft
