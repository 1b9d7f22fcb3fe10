// S1 projection (angl2proj, src/module_energy_cproj_mrso.f90:276-290) on CUDA cores, as a
// persistent pipeline: each resident CTA walks the 64-point tiles blockIdx.x,
// +gridDim.x, ...  Thread 0 issues one bulk copy of the tile's xi (64 x no FP32,
// contiguous) into one of two shared-memory stages, so the next tile is in flight while the
// current one is computed.  Each tile is converted once into drho = rho0 (xi^2 - 1),
// formed in FP64 and rounded, transposed to [io][point] so that a lane reads its own point's values
// without bank conflicts.  The matrix A (no x 2np) stays in shared memory for the launch.
//
// Warp w owns projections 4w..4w+3 (8 real columns, read as two broadcast vector loads per
// io) and lane l the points l and l+32, so each plane store is a coalesced 256-byte
// run.  Used when N is a multiple of 64, np <= 32 (mmax <= 3), xi is 16-byte aligned and
// the stages fit: the FP32 phase of a mixed solve where the tensor-core forms do not apply.
#pragma once

#include "common.cuh"
#include "k_angular.cuh"
#include "k_fft.cuh"
#include "k_tma.cuh"

namespace mdft {

constexpr int kPtBM = 64;      // points per tile
constexpr int kPtStages = 2;
constexpr int kPtLd = kPtBM + 1;  // padded row of the transposed tile

inline int pt_warps(int np) { return (np + 3) / 4; }
inline size_t project_tma_smem_bytes(int np, int no) {
    const size_t a = (size_t)no * 8 * pt_warps(np) * sizeof(float);
    const size_t dr = ((size_t)no * kPtLd * sizeof(float) + 15) / 16 * 16;
    const size_t st = (size_t)kPtBM * no * sizeof(float);
    return (a + 15) / 16 * 16 + dr + kPtStages * st;
}

__global__ void __launch_bounds__(256, 2) k_project_tma(const float *__restrict__ xi, const float *__restrict__ A, float2 *__restrict__ planes,
                                                        int *__restrict__ err, AngularArgs a, int ntiles) {
    const int no = a.no, np = a.np;
    const int nw = (np + 3) / 4, NC = 8 * nw;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    extern __shared__ __align__(128) unsigned char pt_smem[];
    float *As = reinterpret_cast<float *>(pt_smem);  // [no][NC]
    float *dr = reinterpret_cast<float *>(pt_smem + ((size_t)no * NC * sizeof(float) + 15) / 16 * 16);  // [no][kPtLd]
    unsigned char *stage0 = reinterpret_cast<unsigned char *>(dr) + ((size_t)no * kPtLd * sizeof(float) + 15) / 16 * 16;
    const size_t sbytes = (size_t)kPtBM * no * sizeof(float);
    __shared__ uint64_t full[kPtStages];
    __shared__ int abort_flag;
    const int nmine = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

    auto issue = [&](int i) {  // thread 0
        const int s = i % kPtStages;
        const long long pt0 = (long long)((int)blockIdx.x + i * (int)gridDim.x) * kPtBM;
        mbar_arrive_expect_tx(&full[s], (uint32_t)sbytes);
        bulk_load(stage0 + s * sbytes, xi + pt0 * no, (uint32_t)sbytes, &full[s]);
    };
    if (tid == 0) {
        for (int s = 0; s < kPtStages; ++s) mbar_init(&full[s], 1);
        mbar_fence_init();
        abort_flag = 0;
        for (int i = 0; i < kPtStages && i < nmine; ++i) issue(i);
    }
    for (int f = tid; f < no * NC; f += blockDim.x) {
        const int io = f / NC, j = f % NC;
        As[f] = j < 2 * np ? A[(size_t)io * 2 * np + j] : 0.0f;
    }
    __syncthreads();

    for (int i = 0; i < nmine; ++i) {
        const int s = i % kPtStages;
        const bool ok = mbar_wait(&full[s], (uint32_t)((i / kPtStages) & 1));
        if (!ok) abort_flag = 1;
        if (ok) {
            const float *xs = reinterpret_cast<const float *>(stage0 + s * sbytes);
            for (int e = tid; e < kPtBM * no; e += blockDim.x) {
                const int p = e / no, io = e % no;
                const double x = (double)xs[e];
                dr[io * kPtLd + p] = (float)(a.rho0 * (x * x - 1.0));
            }
        }
        __syncthreads();  // transposed tile ready, stage s consumed
        if (abort_flag) break;
        if (tid == 0 && i + kPtStages < nmine) issue(i + kPtStages);
        if (warp < nw) {
            float acc[2][8];
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[p][j] = 0.0f;
            const float *ar = As + 8 * warp;
#pragma unroll 4
            for (int io = 0; io < no; ++io) {
                const float d0 = dr[io * kPtLd + lane], d1 = dr[io * kPtLd + lane + 32];
                const float4 *br = reinterpret_cast<const float4 *>(ar + (size_t)io * NC);
                const float4 b0 = br[0], b1 = br[1];
                const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    acc[0][j] = fma(d0, b[j], acc[0][j]);
                    acc[1][j] = fma(d1, b[j], acc[1][j]);
                }
            }
            const long long pt0 = (long long)((int)blockIdx.x + i * (int)gridDim.x) * kPtBM;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int ip = 4 * warp + q;
                if (ip >= np) break;
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    planes[(size_t)ip * a.N + pt0 + lane + 32 * p] = make_float2(acc[p][2 * q], acc[p][2 * q + 1]);
                }
            }
        }
        __syncthreads();  // the transposed tile is free for the next one
    }
    if (abort_flag && tid == 0) {
        atomicExch(err, 1);
        for (int i = 0; i < nmine; ++i)
            if (!mbar_try_wait(&full[i % kPtStages], (uint32_t)((i / kPtStages) & 1))) {
                (void)mbar_wait(&full[i % kPtStages], (uint32_t)((i / kPtStages) & 1));
                if (i + 1 < nmine) (void)mbar_wait(&full[(i + 1) % kPtStages], (uint32_t)(((i + 1) / kPtStages) & 1));
                break;
            }
    }
}

}  // namespace mdft
