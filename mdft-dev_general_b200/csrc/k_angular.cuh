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

// Sum n rows of kGatherSums partials into out[0..5] (one block, fixed order): entry 4 is a
// maximum, the others sums.
__global__ void k_reduce_sums(const double *__restrict__ partial, long long n, double *__restrict__ out) {
    __shared__ double s[kGatherSums][256];
    double a[kGatherSums] = {0, 0, 0, 0, 0, 0};
    for (long long i = threadIdx.x; i < n; i += blockDim.x) {
        const double *pp = partial + kGatherSums * i;
        for (int j = 0; j < kGatherSums; ++j) a[j] = j == 4 ? fmax(a[j], pp[j]) : a[j] + pp[j];
    }
    for (int j = 0; j < kGatherSums; ++j) s[j][threadIdx.x] = a[j];
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1) {
        if ((int)threadIdx.x < off) {
            for (int j = 0; j < kGatherSums; ++j)
                s[j][threadIdx.x] = j == 4 ? fmax(s[j][threadIdx.x], s[j][threadIdx.x + off]) : s[j][threadIdx.x] + s[j][threadIdx.x + off];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int j = 0; j < kGatherSums; ++j) out[j] = s[j][0];
}

}  // namespace mdft
