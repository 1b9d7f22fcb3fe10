// C-ABI of the B200 MDFT engine (declared in include/mdft_b200.h).
#include "../../include/mdft_b200.h"

#include <algorithm>
#include <cmath>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <atomic>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <string>
#include <thread>

#include "common.cuh"
#include "setup_host.cuh"
#include "k_angular.cuh"
#include "k_fft.cuh"
#include "k_fft3.cuh"
#include "k_oz.cuh"
#include "k_oz2.cuh"
#include "k_ozc.cuh"
#include "k_vec.cuh"
#include "k_lbfgs.cuh"
#include "k_gather_tma.cuh"
#include "k_ozp.cuh"
#include "k_project_tma.cuh"
#include "k_angular_mma.cuh"
#include "k_angular_umma.cuh"
#include "k_vext.cuh"
#include "k_bridge.cuh"

namespace mdft {

static thread_local std::string g_error;
void set_error(const char *fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_error = buf;
}
const char *last_error() { return g_error.c_str(); }

constexpr double kBoltz = 1.3806488e-23;  // src/module_constants.f90:26
constexpr double kNavo = 6.02214129e23;   // src/module_constants.f90:24

enum Stage { ST_PROJECT = 0, ST_FFT_FWD, ST_OZ, ST_FFT_INV, ST_GATHER, ST_COUNT };

struct FftAxis {
    FftAxisArgs args;
    size_t smem;
};

}  // namespace mdft

using namespace mdft;

struct mdft_handle {
    Grid g;
    // set on species 0's handle while mdft_mixture_minimize runs: the minimiser's vectors
    // span every species and its evaluations are the mixture's
    mdft_mixture *mix = nullptr;
    CTable ct;
    int precision = MDFT_PREC_FP64;
    int device = 0;
    cudaStream_t stream = nullptr;
    double const_corr = 0.0;
    bool have_vext = false;
    // device state
    DevBuf<double> xi, vext, df, w, A, B, partial, sums;
    DevBuf<float> vext32;  // FP32 copy of vext for the FP32 phase of mixed solves (made per solve)
    DevBuf<double2> planes, ctab;
    DevBuf<double2> tw64[3];
    // mixed path: FP32 projections, c table, twiddles and angular matrices
    DevBuf<float> A32, B32;
    DevBuf<float2> planes32, ctab32, tw32[3];
    int eval_prec = MDFT_PREC_FP64;  // precision of the evaluations run_pipeline performs
    double *h_sums = nullptr;  // pinned copy of sums; [6..7]: of the last evaluation with a bridge, 0 without
    int nsm = 148;
    // angular transforms of FP64 evaluations [0], and of FP32 ones outside the tensor-core forms
    // [1] (k_project_mma, k_gather_mma), with their matrix images
    DmShape dm_p[2], dm_g[2];
    DevBuf<double2> dm_pimg[2], dm_gimg[2], dm_log;
    int gt_ncol32 = 0;      // k_gather_tma columns of 32 (0: not usable)
    bool pt_ok32 = false;   // k_project_tma usable
    int pt_grid_x32 = 0;                    // resident CTAs of k_project_tma
    DevBuf<int> kerr;                  // set by a pipeline kernel whose bounded wait ran out; [1]: gather CTAs done
    int *h_kerr = nullptr;
    FftAxis fft[3];
    Oz2Args oz{};
    DevBuf<int> oz_ints;
    DevBuf<double> oz_dbls;
    // OZ of every evaluation (k_ozc): the c table by chi block and the cells' records
    OzcArgs ozc{};
    bool ozc_ok = false;  // mrso 2, or mmax 0 where all are alike; k_oz2 otherwise
    DevBuf<int> ozc_xu;  // recursion of the records
    DevBuf<double> ozc_cf, ozc_rec64;
    DevBuf<float> ozc_rec32;
    DevBuf<double2> ozc_c64;
    DevBuf<float2> ozc_c32;
    int oz_warps[2] = {8, 8}, oz_grid[2] = {0, 0};  // k_oz2<double>, k_oz2<float>
    size_t oz_smem[2] = {0, 0};
    int ozc_grid64 = 0, ozc_grid32 = 0;
    // FP32 evaluations: angular contractions on the tensor cores (k_project_umma,
    // k_gather_umma), with the packed split-BF16 images of A^T and B^T
    bool um_ok = false;
    UmmaShape um_ps{}, um_gs{};
    DevBuf<uint16_t> um_pimg, um_gimg;
    int um_grid_p = 0, um_grid_g = 0;
    bool ring_p = false, ring_g = false;  // FP32 phase: the bulk-copy ring forms (one CTA per SM)
    bool ring_p_ok = false, ring_g_ok = false;  // ... where they fit
    // autotuning of the FP32 forms (project: register/ring, OZ: factored/unfactored, gather:
    // ring/register), once per handle on its first FP32 phase; tune_ms[stage][config] are the
    // measured stage times of the two configurations timed (-1: not measured)
    bool tune_on = false, tuned = false;
    double tune_ms[3][2] = {{-1, -1}, {-1, -1}, {-1, -1}};
    bool ozp_ok = false;  // the thread-per-pair k_ozp exists for this order
    bool ozd = false;     // FP32 evaluations with factored rotations, k_ozc (MDFT_OZ=ozp: k_ozp)
    OzpParams ozp{};
    DevBuf<float2> ozp_cq;  // c interpolated at every |q|^2 of a cubic grid (empty: interpolate per pair)
    bool fp32_ok = false, ozp_cq_ok = false;  // ensure_fp32, ensure_ozp_cq have run
    // timing
    bool timing = false;
    bool trace = false;  // MDFT_TRACE=1 in the environment at create: per-iteration log on stderr
    cudaEvent_t ev[ST_COUNT + 1] = {};
    double stage_ms[ST_COUNT] = {0};
    int stage_count = 0;
    long long launches = 0;  // kernels launched by this handle
    // the evaluation pipeline as CUDA graphs, one per set of buffers and flags (MDFT_GRAPHS=0:
    // direct launches); never used while stage timing is on
    struct PipeGraph {
        const void *x, *dvec, *vext, *vext32;
        double *g;
        int do_ideal, df_mode, prec;
        bool v32, x32;
        cudaGraphExec_t exec;
        long long nlaunch;
    };
    std::vector<PipeGraph> pipe_graphs;
    bool graphs_on = true;
    bool wait_fail = false;  // mdft_set_wait_failure: gathers report a timed-out wait (tests)
    // vector reductions
    DevBuf<double> vpart, vsc;
    double *h_vsc = nullptr;
    // minimiser work (allocated on first use)
    LbfgsState lb;
    // learned warm start (mdft_set_warm_net): the network, its input channels, the
    // orientation table {u_x, u_y, u_z, w} and the solute sites, allocated on first use
    mdft_warm_net *warm = nullptr;
    DevBuf<float> wfeat;
    DevBuf<double4> wdir;
    DevBuf<double> wsite;
    long long warm_starts = 0, warm_fallbacks = 0;
    // bridge = "cgb" (mdft_set_bridge_cgb): 0 none, 1 'sla', 2 'wda'; the transformed kernel,
    // two work planes, n(r) and the block partials
    int cgb = 0;
    CgbArgs cgb_args{};
    DevBuf<double2> cgb_kk, cgb_a, cgb_b;
    DevBuf<double> cgb_dens, cgb_part;
    // bridge = "hard_sphere" (mdft_set_bridge_fmt): 0 none, 1 PY, 2 CS; seven work planes,
    // the hard-sphere c(k) and the partials {density 2B | stats 2 | Phi 4B | gradient 4B}
    int fmt = 0;
    FmtArgs fmt_args{};
    DevBuf<double2> fmt_pl;
    DevBuf<double> fmt_cs, fmt_part;
};

namespace {
bool has_bridge(const mdft_handle *h) { return h->cgb || h->fmt; }
}

namespace {

int check_cuda(cudaError_t e, const char *what) {
    if (e != cudaSuccess) {
        set_error("%s: %s", what, cudaGetErrorString(e));
        return MDFT_E_CUDA;
    }
    return 0;
}

int alloc_check(cudaError_t e, const char *what, size_t bytes) {
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        set_error("device allocation of %zu bytes for %s failed", bytes, what);
        return MDFT_E_NOMEM;
    }
    return check_cuda(e, what);
}

// Let `fn` use all opt-in shared memory that its static allocation leaves.
int allow_smem(const void *fn, int optin) {
    cudaFuncAttributes at{};
    int rc = check_cuda(cudaFuncGetAttributes(&at, fn), "cudaFuncGetAttributes");
    if (rc) return rc;
    return check_cuda(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)at.sharedSizeBytes),
                      "cudaFuncSetAttribute");
}

int upload_twiddles(DevBuf<double2> &buf, int n) {
    std::vector<double2> h(n);
    for (int t = 0; t < n; ++t) {
        long double ang = 2.0L * 3.141592653589793238462643383279502884L * (long double)t / (long double)n;
        h[t] = make_double2((double)cosl(ang), (double)sinl(ang));
    }
    int rc = alloc_check(buf.alloc(n), "fft twiddles", n * sizeof(double2));
    if (rc) return rc;
    return check_cuda(cudaMemcpy(buf.p, h.data(), n * sizeof(double2), cudaMemcpyHostToDevice), "twiddle upload");
}

// BF16 bits of an FP32 value, rounded to nearest even (finite inputs)
uint16_t bf16_bits(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    u += 0x7FFFu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}
float bf16_value(uint16_t b) {
    const uint32_t u = (uint32_t)b << 16;
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
// hi and lo BF16 images (hi then lo) of an [Rp][Kp] operand in the packed tcgen05 layout;
// value(r, k) is the FP64 entry (0 in the padding)
template <typename F>
void pack_split_bf16(int Rp, int Kp, F value, std::vector<uint16_t> &img) {
    const size_t half = (size_t)Rp * Kp;
    img.assign(2 * half, 0);
    for (int r = 0; r < Rp; ++r)
        for (int k = 0; k < Kp; ++k) {
            const double v = value(r, k);
            const uint16_t hi = bf16_bits((float)v);
            const uint16_t lo = bf16_bits((float)(v - (double)bf16_value(hi)));
            const size_t off = umma::elem_offset(r, k, Kp, 2) / 2;
            img[off] = hi;
            img[half + off] = lo;
        }
}

int pick_tl(long long lines_divisor, int n) {
    int best = 1;
    const int cands[] = {32, 16, 8, 4, 2, 1};
    for (int c : cands) {
        if (lines_divisor % c) continue;
        if (c == 32 && n > 32) continue;
        best = c;
        break;
    }
    return best;
}

int setup_fft(mdft_handle *h) {
    const Grid &g = h->g;
    const int dims[3] = {g.nx, g.ny, g.nz};
    for (int ax = 0; ax < 3; ++ax) {
        FftAxis &F = h->fft[ax];
        F.args.axis = ax;
        F.args.nx = g.nx;
        F.args.ny = g.ny;
        F.args.nz = g.nz;
        F.args.nplanes = g.np;
        if (!make_plan1d(dims[ax], F.args.plan)) {
            set_error("grid size %d is not of the form 2^a 3^b", dims[ax]);
            return MDFT_E_ARG;
        }
        long long lines_div = (ax == 0) ? (long long)g.np * g.ny * g.nz : g.nx;
        F.args.TL = pick_tl(lines_div, dims[ax]);
        F.smem = fft_smem_bytes<double>(dims[ax], F.args.TL);
        int rc = upload_twiddles(h->tw64[ax], dims[ax]);
        if (rc) return rc;
        std::vector<double2> t64(dims[ax]);
        cudaMemcpy(t64.data(), h->tw64[ax].p, dims[ax] * sizeof(double2), cudaMemcpyDeviceToHost);
        std::vector<float2> t32(dims[ax]);
        for (int t = 0; t < dims[ax]; ++t) t32[t] = make_float2((float)t64[t].x, (float)t64[t].y);
        if ((rc = alloc_check(h->tw32[ax].alloc(dims[ax]), "fft twiddles", dims[ax] * sizeof(float2)))) return rc;
        cudaMemcpy(h->tw32[ax].p, t32.data(), dims[ax] * sizeof(float2), cudaMemcpyHostToDevice);
    }
    return 0;
}

// A pipeline kernel behind another one of the pipeline in the stream.  On small grids with
// programmatic dependent launch, which hides launch and set-up (16^3 mmax 1: 33.8 -> 30.4 us an
// evaluation); not on large ones, where the next kernel's CTAs take room from the running one's
// (64^3 mmax 3 FP64: 635 -> 706 us, FP32: 518 -> 528; 32^3 mmax 5, 46 MB of planes: even).
// All kernels launched here call pdl_wait in every CTA.
constexpr size_t kPdlMostBytes = 16u << 20;
cudaError_t launch_pipe(const mdft_handle *h, const void *fn, unsigned grid, unsigned block, void **args, size_t smem) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = h->stream;
    c.attrs = &at;
    c.numAttrs = (size_t)h->g.np * h->g.N * 16 <= kPdlMostBytes ? 1 : 0;
    return cudaLaunchKernelExC(&c, fn, args);
}
SumsOut sums_out(mdft_handle *h) {
    return SumsOut{h->sums.p, h->h_sums, h->kerr.p, h->h_kerr, reinterpret_cast<unsigned *>(h->kerr.p + 1)};
}

// The transforms of one length and direction: whole planes (null where a plane does not fit in
// shared memory), lines, columns.
struct FftFns {
    const void *xy = nullptr, *lines = nullptr, *cols = nullptr;
    size_t xy_smem = 0, lines_smem = 0, cols_smem = 0;
    int xy_threads = 0, cols_threads = 0;
};
template <typename T, int N, int S>
FftFns fft_fns_n() {
    FftFns f;
    if constexpr (fft_xy_fits<T, N>()) {
        f.xy = (const void *)k_fft_xy<T, N, S>;
        f.xy_smem = fft_xy_smem<T, N>();
        f.xy_threads = fft_xy_threads<T, N>();
    }
    f.lines = (const void *)k_fft_lines<T, N, S>;
    f.lines_smem = fft_lines_smem<T, N>();
    f.cols = (const void *)k_fft_cols<T, N, S>;
    f.cols_smem = fft_cols_smem<T, N>();
    f.cols_threads = fft_col_threads<T, N>();
    return f;
}
// lines == null: no kernel for this length (k_fft_axis covers it)
template <typename T, int S>
FftFns fft_fns_s(int n) {
    switch (n) {
        case 8: return fft_fns_n<T, 8, S>();
        case 12: return fft_fns_n<T, 12, S>();
        case 16: return fft_fns_n<T, 16, S>();
        case 18: return fft_fns_n<T, 18, S>();
        case 24: return fft_fns_n<T, 24, S>();
        case 32: return fft_fns_n<T, 32, S>();
        case 36: return fft_fns_n<T, 36, S>();
        case 48: return fft_fns_n<T, 48, S>();
        case 54: return fft_fns_n<T, 54, S>();
        case 64: return fft_fns_n<T, 64, S>();
        case 72: return fft_fns_n<T, 72, S>();
        case 96: return fft_fns_n<T, 96, S>();
        case 128: return fft_fns_n<T, 128, S>();
    }
    return FftFns();
}
template <typename T>
FftFns fft_fns(int n, int sign) { return sign > 0 ? fft_fns_s<T, 1>(n) : fft_fns_s<T, -1>(n); }

template <typename T>
int setup_fft_smem(int n, int maxsmem) {
    int rc;
    for (int sign : {1, -1}) {
        const FftFns f = fft_fns<T>(n, sign);
        for (const void *fn : {f.xy, f.lines, f.cols})
            if (fn && (rc = allow_smem(fn, maxsmem))) return rc;
    }
    return 0;
}

// 3-D FFT of nplanes planes on the handle's grid, in place.
template <typename T>
int launch_fft_t(mdft_handle *h, typename Cplx<T>::t *data, long long nplanes, int sign) {
    using C = typename Cplx<T>::t;
    const Grid &g = h->g;
    const int dims[3] = {g.nx, g.ny, g.nz};
    const long long nxy = (long long)g.nx * g.ny;
    const C *tw[3];
    for (int ax = 0; ax < 3; ++ax) tw[ax] = sizeof(T) == 8 ? (const C *)h->tw64[ax].p : (const C *)h->tw32[ax].p;
    cudaError_t e = cudaSuccess;
    const FftFns fx = fft_fns<T>(g.nx, sign);
    int first = 0;
    if (g.nx == g.ny && fx.xy) {
        void *args[] = {(void *)&data, (void *)&tw[0]};
        e = launch_pipe(h, fx.xy, (unsigned)(nplanes * g.nz), fx.xy_threads, args, fx.xy_smem);
        h->launches += 1;
        first = 2;
    }
    for (int ax = first; ax < 3 && e == cudaSuccess; ++ax) {
        const FftFns f = ax == 0 ? fx : fft_fns<T>(dims[ax], sign);
        h->launches += 1;
        if (!f.lines) {
            FftAxisArgs a = h->fft[ax].args;
            a.nplanes = nplanes;
            a.sign = sign;
            a.TL = pick_tl(ax == 0 ? nplanes * g.ny * g.nz : g.nx, dims[ax]);
            const long long nlines = nplanes * g.N / dims[ax];
            k_fft_axis<T><<<(unsigned)(nlines / a.TL), kFftThreads, fft_smem_bytes<T>(dims[ax], a.TL), h->stream>>>(data, tw[ax], a);
            e = cudaGetLastError();
        } else if (ax == 0) {
            long long nlines = nplanes * g.ny * g.nz;
            void *args[] = {(void *)&data, (void *)&tw[0], (void *)&nlines};
            e = launch_pipe(h, f.lines, (unsigned)((nlines + kFftLines - 1) / kFftLines), kFftLineThreads, args, f.lines_smem);
        } else {
            long long ncol = ax == 1 ? nplanes * g.nz * g.nx : nplanes * nxy, outer = ax == 1 ? nxy : g.N, es = ax == 1 ? g.nx : nxy;
            unsigned inner = ax == 1 ? (unsigned)g.nx : (unsigned)nxy;
            void *args[] = {(void *)&data, (void *)&tw[ax], (void *)&ncol, (void *)&inner, (void *)&outer, (void *)&es};
            e = launch_pipe(h, f.cols, (unsigned)((ncol + fft_cols<T>() - 1) / fft_cols<T>()), f.cols_threads, args, f.cols_smem);
        }
    }
    return check_cuda(e, "fft launch");
}

// FP32 OZ, thread per pair: the instantiation for (mmax, mrso); the c(k) layouts hold mrso 1 at
// mmax 0 only
const void *ozp_kernel(int mmax, int mrso) {
    switch (10 * mrso + mmax) {
        case 20: return (const void *)k_ozp<0, 2>;
        case 21: return (const void *)k_ozp<1, 2>;
        case 22: return (const void *)k_ozp<2, 2>;
        case 23: return (const void *)k_ozp<3, 2>;
        case 10: return (const void *)k_ozp<0, 1>;
    }
    return nullptr;
}
void launch_ozp(mdft_handle *h, float2 *planes, const float2 *ctab, const Oz2Args &oz) {
    const Grid &g = h->g;
    const unsigned grid = (unsigned)((oz.nk + kOzpThreads - 1) / kOzpThreads);
    const size_t smem = ozp_smem_bytes(g.np);
    const float2 *cq = h->ozp_cq.p;
    void *args[] = {(void *)&planes, (void *)&ctab, (void *)&oz, (void *)&h->ozp, (void *)&cq};
    cudaLaunchKernel(ozp_kernel(g.mmax, g.mrso), dim3(grid), dim3(kOzpThreads), args, smem, h->stream);
}

// k_ozc for an angular order
template <typename T>
const void *ozc_kernel(int mmax) {
    switch (mmax) {
        case 0: return (const void *)k_ozc<T, 0>;
        case 1: return (const void *)k_ozc<T, 1>;
        case 2: return (const void *)k_ozc<T, 2>;
        case 3: return (const void *)k_ozc<T, 3>;
        case 4: return (const void *)k_ozc<T, 4>;
        default: return (const void *)k_ozc<T, 5>;
    }
}
// In-place OZ step of one species on planes.
template <typename T>
void launch_oz(mdft_handle *h, typename Cplx<T>::t *planes) {
    const bool dbl = sizeof(T) == 8;
    if (!h->ozc_ok) {
        Oz2Args oz = h->oz;
        oz.quirks = dbl ? 1 : 0;
        const typename Cplx<T>::t *ctab = dbl ? (const typename Cplx<T>::t *)h->ctab.p : (const typename Cplx<T>::t *)h->ctab32.p;
        k_oz2<T><<<h->oz_grid[!dbl], 32 * h->oz_warps[!dbl], h->oz_smem[!dbl], h->stream>>>(planes, ctab, h->oz_ints.p, h->oz_dbls.p, oz,
                                                                                            nullptr, OzMix{});
        return;
    }
    OzcArgs a = h->ozc;
    a.quirks = dbl ? 1 : 0;
    const void *c = dbl ? (const void *)h->ozc_c64.p : (const void *)h->ozc_c32.p;
    const void *rec = dbl ? (const void *)h->ozc_rec64.p : (const void *)h->ozc_rec32.p;
    void *args[] = {(void *)&planes, (void *)&c, (void *)&rec, (void *)&a};
    const int M = h->g.mmax;
    launch_pipe(h, ozc_kernel<T>(M), dbl ? h->ozc_grid64 : h->ozc_grid32, 32 * ozc_warps(M), args, ozc_smem_bytes<T>(M));
}
// Tables and launch shape of k_ozc<T>.
template <typename T>
int setup_ozc(mdft_handle *h, const std::vector<double> &cx, DevBuf<typename Cplx<T>::t> &ctab, DevBuf<T> &rec, int &grid, int maxsmem) {
    const Grid &g = h->g;
    const std::vector<T> c(cx.begin(), cx.end());
    const size_t nrec = (size_t)h->ozc.ncell * ozc_rec(g.mmax);
    int rc;
    if ((rc = alloc_check(ctab.alloc(c.size() / 2), "c table", c.size() * sizeof(T)))) return rc;
    cudaMemcpy(ctab.p, c.data(), c.size() * sizeof(T), cudaMemcpyHostToDevice);
    if ((rc = alloc_check(rec.alloc(nrec), "OZ cell records", nrec * sizeof(T)))) return rc;
    const OzcSetup su{h->ozc.hx, h->ozc.hy, h->ozc.ncell, g.mmax, sizeof(T) == 8 ? 1 : 0, h->ct.dq, 2.0 * kPi / g.lx, 2.0 * kPi / g.ly,
                      2.0 * kPi / g.lz};
    // the uploads have reached the device (the handle's stream does not wait for the legacy one)
    if ((rc = check_cuda(cudaStreamSynchronize(cudaStreamLegacy), "OZ tables"))) return rc;
    k_ozc_records<T><<<(h->ozc.ncell + 3) / 4, 128, 0, h->stream>>>(rec.p, h->ozc_xu.p, h->ozc_cf.p, su);
    if ((rc = check_cuda(cudaGetLastError(), "OZ cell records"))) return rc;
    const void *fn = ozc_kernel<T>(g.mmax);
    if ((rc = allow_smem(fn, maxsmem))) return rc;
    // persistent: as many CTAs as fit on the device at once
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 32 * ozc_warps(g.mmax), ozc_smem_bytes<T>(g.mmax));
    grid = std::min((h->ozc.ncell + kOzcCells - 1) / kOzcCells, std::max(1, per_sm) * h->nsm);
    return 0;
}

void stage_mark(mdft_handle *h, int i) {
    if (h->timing) cudaEventRecord(h->ev[i], h->stream);
}

// Arguments of the S7 gather.  The excess prefactor -kT 2 (4 pi^2) / mrso / n0
// (src/module_energy_cproj_mrso.f90:728) carries a species' mole fraction as `scale` in a
// multi-species evaluation (src/module_energy_cproj_mrso_mixture.f90:791).
GatherArgs gather_args(const mdft_handle *h, int df_mode, int do_ideal, const void *dvec, double scale) {
    const Grid &g = h->g;
    GatherArgs ga;
    ga.fail_wait = h->wait_fail ? 1 : 0;
    ga.N = g.N;
    ga.no = g.no;
    ga.np = g.np;
    ga.rho0 = g.rho0;
    ga.kT = g.kT;
    ga.dv = g.dv;
    const double fourpisq = 4.0 * kPi * kPi;
    ga.prefactor = -g.kT * 2.0 * fourpisq / g.mrso / g.n0;
    if (scale != 1.0) ga.prefactor *= scale;
    ga.cst = 1.0 / (double)(g.nx * g.ny * g.nz);
    ga.do_ideal = do_ideal;
    ga.df_mode = df_mode;
    ga.dvec = dvec;
    return ga;
}

int launch_fft_planes(mdft_handle *h, double2 *data, int nplanes, int sign) { return launch_fft_t<double>(h, data, nplanes, sign); }

// The bridge term after the pipeline of a full FP64 evaluation: F_b into sums[6]; with d_df,
// the bridge gradient added to d_df and sums[3..5] recomputed over the final gradient.
int launch_fmt(mdft_handle *h, const double *d_xi, double *d_df, const double *dvec) {
    const FmtArgs &a = h->fmt_args;
    const unsigned nb = kRedBlocks;
    const long long N = h->g.N;
    double2 *pl = h->fmt_pl.p;
    double *pd = h->fmt_part.p, *stats = pd + 2 * nb, *pphi = stats + 2, *pgr = pphi + 4 * nb;
    int rc;
    k_fmt_density<<<nb, kBrThreads, 0, h->stream>>>(d_xi, h->w.p, a, pl, pd);
    k_fmt_stats<<<1, kBrThreads, 0, h->stream>>>(pd, (int)nb, stats);
    if ((rc = launch_fft_planes(h, pl, 2, -1))) return rc;
    k_fmt_weigh<<<nb, kBrThreads, 0, h->stream>>>(pl, h->fmt_cs.p, a);
    if ((rc = launch_fft_planes(h, pl + N, 5, +1))) return rc;
    k_fmt_phi<<<nb, kBrThreads, 0, h->stream>>>(pl, a, d_df ? 1 : 0, pphi);
    h->launches += 4;
    if (d_df) {
        if ((rc = launch_fft_planes(h, pl + 2 * N, 4, -1))) return rc;
        k_fmt_combine<<<nb, kBrThreads, 0, h->stream>>>(pl, a);
        if ((rc = launch_fft_planes(h, pl + 6 * N, 1, +1))) return rc;
        h->launches += 1;
    }
    k_fmt_grad<<<nb, kBrThreads, 0, h->stream>>>(d_xi, h->w.p, a, pl, stats, d_df, dvec, pgr);
    k_fmt_finish<<<1, kBrThreads, 0, h->stream>>>(pphi, pgr, (int)nb, stats, a, d_df ? 1 : 0, h->sums.p);
    k_publish_sums<<<1, 32, 0, h->stream>>>(sums_out(h), 3, 8);
    h->launches += 3;
    return check_cuda(cudaGetLastError(), "bridge launch");
}

int launch_bridge(mdft_handle *h, const double *d_xi, double *d_df, const double *dvec) {
    if (h->fmt) return launch_fmt(h, d_xi, d_df, dvec);
    const Grid &g = h->g;
    const CgbArgs &a = h->cgb_args;
    const unsigned nb = kRedBlocks;
    int rc;
    k_cgb_density<<<nb, kBrThreads, 0, h->stream>>>(d_xi, h->w.p, a, h->cgb_dens.p, h->cgb_a.p);
    if ((rc = launch_fft_planes(h, h->cgb_a.p, 1, -1))) return rc;
    k_cgb_cmul<<<nb, kBrThreads, 0, h->stream>>>(h->cgb_a.p, h->cgb_kk.p, g.N);
    if ((rc = launch_fft_planes(h, h->cgb_a.p, 1, +1))) return rc;
    k_cgb_phi<<<nb, kBrThreads, 0, h->stream>>>(h->cgb_a.p, h->cgb_dens.p, a, d_df ? 1 : 0, h->cgb_b.p, h->cgb_part.p);
    h->launches += 4;
    if (d_df) {
        if ((rc = launch_fft_planes(h, h->cgb_b.p, 1, -1))) return rc;
        k_cgb_cmul<<<nb, kBrThreads, 0, h->stream>>>(h->cgb_b.p, h->cgb_kk.p, g.N);
        if ((rc = launch_fft_planes(h, h->cgb_b.p, 1, +1))) return rc;
        k_cgb_grad<<<nb, kBrThreads, 0, h->stream>>>(d_xi, h->w.p, a, h->cgb_a.p, h->cgb_b.p, h->cgb_dens.p, d_df, dvec,
                                                     h->cgb_part.p + kRedBlocks);
        h->launches += 2;
    }
    k_cgb_finish<<<1, kBrThreads, 0, h->stream>>>(h->cgb_part.p, kRedBlocks, h->cgb_part.p + kRedBlocks, d_df ? kRedBlocks : 0,
                                                  h->sums.p);
    k_publish_sums<<<1, 32, 0, h->stream>>>(sums_out(h), 3, 8);
    h->launches += 2;
    return check_cuda(cudaGetLastError(), "bridge launch");
}

// The kernel of a (WN, NT) shape out of a family F<WN, NT>::fn().
template <template <int, int> class F>
const void *dm_kernel(const DmShape &s) {
    switch (10 * s.wn + s.nt) {
        case 11: return F<1, 1>::fn();
        case 12: return F<1, 2>::fn();
        case 22: return F<2, 2>::fn();
        case 42: return F<4, 2>::fn();
        case 43: return F<4, 3>::fn();
        default: return F<4, 4>::fn();
    }
}
template <typename T, int ROWS> struct DmProject {
    template <int WN, int NT> struct F { static const void *fn() { return (const void *)&k_project_mma<T, WN, NT, ROWS>; } };
};
template <typename T, bool V16, typename TD> struct DmGather {
    template <int WN, int NT> struct F { static const void *fn() { return (const void *)&k_gather_mma<T, WN, NT, V16, TD>; } };
};
template <typename T> const void *project_mma_fn(const DmShape &s, int rows) {
    return rows == kRowEven  ? dm_kernel<DmProject<T, kRowEven>::template F>(s)
           : rows == kRowOdd ? dm_kernel<DmProject<T, kRowOdd>::template F>(s)
                             : dm_kernel<DmProject<T, kRowAny>::template F>(s);
}
template <typename T> const void *gather_mma_fn(const DmShape &s, bool v16, bool v32) {
    return v32 ? (v16 ? dm_kernel<DmGather<T, true, float>::template F>(s) : dm_kernel<DmGather<T, false, float>::template F>(s))
               : (v16 ? dm_kernel<DmGather<T, true, double>::template F>(s) : dm_kernel<DmGather<T, false, double>::template F>(s));
}
// Shapes, matrix images and persistent grids of k_project_mma<T>, k_gather_mma<T>.
template <typename T>
int setup_mma(mdft_handle *h, const std::vector<double> &A, const std::vector<double> &B, size_t dyn_max, int maxsmem) {
    const Grid &g = h->g;
    const int i = sizeof(T) == 8 ? 0 : 1, np2 = 2 * g.np, no = g.no;
    DmShape &P = h->dm_p[i], &G = h->dm_g[i];
    P = dm_project_shape<T>(g.np, no, dyn_max);
    G = dm_gather_shape<T>(g.np, no, dyn_max);
    if (!P.nt || !G.nt) { set_error("angular transform tiles do not fit in shared memory"); return MDFT_E_ARG; }
    const std::vector<double2> pi = dm_image<T>(P, [&](int k, int j) { return (k < no && j < np2) ? A[(size_t)k * np2 + j] : 0.0; });
    const std::vector<double2> gi = dm_image<T>(G, [&](int k, int j) { return (k < np2 && j < no) ? B[(size_t)k * no + j] : 0.0; });
    int rc;
    if ((rc = alloc_check(h->dm_pimg[i].alloc(pi.size()), "angular matrices", pi.size() * 16))) return rc;
    if ((rc = alloc_check(h->dm_gimg[i].alloc(gi.size()), "angular matrices", gi.size() * 16))) return rc;
    cudaMemcpy(h->dm_pimg[i].p, pi.data(), pi.size() * 16, cudaMemcpyHostToDevice);
    cudaMemcpy(h->dm_gimg[i].p, gi.data(), gi.size() * 16, cudaMemcpyHostToDevice);
    // resident CTAs, a whole number of column chunks
    auto grid = [&](const DmShape &s, const void *fn, int threads) {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, s.smem);
        const long long tiles = (g.N + s.bm - 1) / s.bm;
        return (int)std::min(tiles, std::max<long long>(1, (long long)std::max(1, per_sm) * h->nsm / s.nchunk)) * s.nchunk;
    };
    for (int rows : {(int)kRowEven, (int)kRowOdd, (int)kRowAny})
        if ((rc = allow_smem(project_mma_fn<T>(P, rows), maxsmem))) return rc;
    for (bool v16 : {false, true}) {
        for (bool v32 : {false, true})
            if ((rc = allow_smem(gather_mma_fn<T>(G, v16, v32), maxsmem))) return rc;
    }
    P.grid = grid(P, project_mma_fn<T>(P, no % 2 == 0 ? kRowEven : kRowOdd), kPmThreads);
    G.grid = grid(G, gather_mma_fn<T>(G, no % 2 == 0, false), kGmThreads);
    return 0;
}

// c rows of k_ozp, when it is first to run (k_ozc needs none).
int ensure_ozp_cq(mdft_handle *h) {
    if (h->ozp_cq_ok || !h->ozp_ok) return 0;
    std::vector<float2> c32(h->ct.c.size() / 2);  // the FP32 table as the kernels read it
    for (size_t i = 0; i < c32.size(); ++i) c32[i] = make_float2((float)h->ct.c[2 * i], (float)h->ct.c[2 * i + 1]);
    const std::vector<float2> cq = build_ozp_cq(h->g, h->ct, c32);
    int rc;
    if (!cq.empty()) {
        if ((rc = alloc_check(h->ozp_cq.alloc(cq.size()), "OZ c rows", cq.size() * 8))) return rc;
        if ((rc = check_cuda(cudaMemcpy(h->ozp_cq.p, cq.data(), cq.size() * 8, cudaMemcpyHostToDevice), "OZ c rows"))) return rc;
    }
    h->ozp_cq_ok = true;
    return 0;
}
bool uses_ozp(const mdft_handle *h) { return h->ozp_ok && !(h->ozd && h->ozc_ok); }

// Tables that only FP32 evaluations read, before the first of them: a mixed handle's creation, or
// the first mixed minimisation of an FP64 handle (which else pays nothing for them).
int ensure_fp32(mdft_handle *h) {
    int rc;
    if (uses_ozp(h) && (rc = ensure_ozp_cq(h))) return rc;
    if (h->fp32_ok) return 0;
    int maxsmem = 0;
    cudaDeviceGetAttribute(&maxsmem, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device);
    std::vector<double> A, B;
    build_angular_matrices(h->g, A, B);
    if ((rc = setup_mma<float>(h, A, B, (size_t)maxsmem - 1024, maxsmem))) return rc;
    if (h->ozc_ok && (rc = setup_ozc<float>(h, build_ozc_table(h->g, h->ct), h->ozc_c32, h->ozc_rec32, h->ozc_grid32, maxsmem))) return rc;
    if ((rc = check_cuda(cudaStreamSynchronize(cudaStreamLegacy), "FP32 tables"))) return rc;
    h->fp32_ok = true;
    return 0;
}

// S1 of an FP64 point.
template <typename T>
void launch_project_mma(mdft_handle *h, const double *d_xi, typename Cplx<T>::t *planes, const AngularArgs &aa) {
    const int i = sizeof(T) == 8 ? 0 : 1;
    const DmShape &s = h->dm_p[i];
    const int rows = ((uintptr_t)d_xi & 15u) != 0 ? kRowAny : h->g.no % 2 == 0 ? kRowEven : kRowOdd;
    const double2 *img = h->dm_pimg[i].p;
    int *err = h->kerr.p;
    DmWalk wk(s, h->g.N);
    void *args[] = {(void *)&d_xi, (void *)&img, (void *)&planes, (void *)&err, (void *)&aa, (void *)&wk};
    launch_pipe(h, project_mma_fn<T>(s, rows), s.grid, kPmThreads, args, s.smem);
}

// S7 + ideal/external of an FP64 point; v32: df and the search direction are FP32 vectors.
// It leaves the evaluation's sums (no k_reduce_sums after it).
template <typename T>
void launch_gather_mma(mdft_handle *h, const typename Cplx<T>::t *planes, const double *d_xi, void *d_df, const GatherArgs &ga, bool v32) {
    const int i = sizeof(T) == 8 ? 0 : 1;
    const DmShape &s = h->dm_g[i];
    auto al = [](const void *p, uintptr_t m) { return ((uintptr_t)p & m) == 0; };
    const uintptr_t m = v32 ? 7u : 15u;
    const bool v16 = h->g.no % 2 == 0 && al(d_xi, 15u) && al(d_df, m) && al(ga.dvec, m);
    const double2 *img = h->dm_gimg[i].p, *lt = h->dm_log.p;
    const double *vext = h->vext.p, *w = h->w.p;
    double *partial = h->partial.p;
    int *err = h->kerr.p;
    DmWalk wk(s, h->g.N);
    SumsOut so = sums_out(h);
    void *args[] = {(void *)&planes, (void *)&img, (void *)&lt, (void *)&d_xi, (void *)&vext, (void *)&w, (void *)&d_df, (void *)&partial, (void *)&err,
                    (void *)&ga, (void *)&wk, (void *)&so};
    launch_pipe(h, gather_mma_fn<T>(s, v16, v32), s.grid, kGmThreads, args, s.smem);
}

// The excess-term pipeline plus (optionally) the ideal/external term on device
// arrays, in precision T; leaves {F_id, F_ext, sum_exc, df.dvec, max|df|} in h->sums.
template <typename T>
int run_pipeline_t(mdft_handle *h, const void *xin, double *d_df, int do_ideal, int df_mode, const void *dvec, bool vec32,
                   bool x32) {
    using C = typename Cplx<T>::t;
    const double *d_xi = static_cast<const double *>(xin);  // FP64 point unless x32
    const Grid &g = h->g;
    const bool dbl = sizeof(T) == 8;
    if (has_bridge(h) && do_ideal && (!dbl || vec32 || x32)) {
        set_error("the bridge term is evaluated in FP64 only (an FP64 handle and FP64 solves)");
        return MDFT_E_STATE;
    }
    C *planes = dbl ? (C *)h->planes.p : (C *)h->planes32.p;
    const T *A = dbl ? (const T *)h->A.p : (const T *)h->A32.p;
    const T *B = dbl ? (const T *)h->B.p : (const T *)h->B32.p;
    const C *ctab = dbl ? (const C *)h->ctab.p : (const C *)h->ctab32.p;
    stage_mark(h, 0);
    AngularArgs aa{g.N, g.no, g.np, g.rho0};
    if (x32 && (dbl || (!h->pt_ok32 && !h->um_ok) || !h->vext32.p || ((uintptr_t)xin & 15u) != 0)) {
        set_error("an FP32 point needs the FP32 bulk-copy kernels");
        return MDFT_E_STATE;
    }
    const bool umma = x32 && h->um_ok;
    if (umma) {
        // FP32 phase of a mixed solve: tensor-core projection (split BF16) of the FP32 point
        const int ntiles = (int)(g.N / kUmBM);
        const unsigned grid = (unsigned)std::min(ntiles, h->um_grid_p);
        const size_t smem = umma_smem_bytes(h->um_ps);
        const bool vec = g.no % 4 == 0 && ((uintptr_t)xin & 15u) == 0;
        if (h->ring_p) {
            const unsigned rgrid = (unsigned)std::min(ntiles, h->nsm);
            const size_t rsmem = project_ring_smem_bytes(h->um_ps, g.no);
            if (vec) k_project_ring<4><<<rgrid, kRingThreads, rsmem, h->stream>>>(static_cast<const float *>(xin), h->um_pimg.p, (float2 *)planes, h->kerr.p, aa, h->um_ps, ntiles);
            else k_project_ring<1><<<rgrid, kRingThreads, rsmem, h->stream>>>(static_cast<const float *>(xin), h->um_pimg.p, (float2 *)planes, h->kerr.p, aa, h->um_ps, ntiles);
        } else {
            if (vec) k_project_umma<4><<<grid, kPjThreads, smem, h->stream>>>(static_cast<const float *>(xin), h->um_pimg.p, (float2 *)planes, h->kerr.p, aa, h->um_ps, ntiles);
            else k_project_umma<1><<<grid, kPjThreads, smem, h->stream>>>(static_cast<const float *>(xin), h->um_pimg.p, (float2 *)planes, h->kerr.p, aa, h->um_ps, ntiles);
        }
    } else if (x32) {
        const int ntiles = (int)(g.N / kPtBM);
        k_project_tma<<<std::min(ntiles, h->pt_grid_x32), 256, project_tma_smem_bytes(g.np, g.no), h->stream>>>(
            static_cast<const float *>(xin), (const float *)A, (float2 *)planes, h->kerr.p, aa, ntiles);
    } else {
        launch_project_mma<T>(h, d_xi, planes, aa);
    }
    int rc = check_cuda(cudaGetLastError(), "project launch");
    if (rc) return rc;
    stage_mark(h, 1);
    if ((rc = launch_fft_t<T>(h, planes, g.np, +1))) return rc;
    stage_mark(h, 2);
    if (!dbl && uses_ozp(h)) launch_ozp(h, (float2 *)planes, (const float2 *)ctab, h->oz);
    else launch_oz<T>(h, planes);
    if ((rc = check_cuda(cudaGetLastError(), "oz launch"))) return rc;
    stage_mark(h, 3);
    if ((rc = launch_fft_t<T>(h, planes, g.np, -1))) return rc;
    stage_mark(h, 4);
    const GatherArgs ga = gather_args(h, d_df ? df_mode : 0, do_ideal, dvec, 1.0);
    const int gt_ncol = h->gt_ncol32;
    auto al16 = [](const void *p) { return ((uintptr_t)p & 15u) == 0; };
    long long red_blocks = 0;
    const bool umma_gather = umma && ga.df_mode != 2;
    if (x32 && !umma_gather && (gt_ncol <= 0 || ga.df_mode == 2 || !al16(dvec))) {
        set_error("an FP32 point needs the bulk-copy gather");
        return MDFT_E_STATE;
    }
    if (umma_gather) {
        // tensor-core gather (split BF16) with the FP32 element-wise epilogue
        const int ntiles = (int)(g.N / kUmBM);
        const int grid = std::min(ntiles, h->um_grid_g);
        const size_t smem = gather_umma_smem_bytes(h->um_gs, g.no);
        const float2 *pl = (const float2 *)planes;
        // 4-element vector epilogue with a compile-time orientation count (mmax 3, water), else scalar
        const bool v84 = g.no == 84 && al16(xin) && al16(dvec) && al16(d_df);
        float *df32 = reinterpret_cast<float *>(d_df);
        const float *x32p = static_cast<const float *>(xin);
        if (v84 && h->ring_g) {
            const int rgrid = std::min(ntiles, h->nsm);
            const size_t rs = gather_ring_smem_bytes(h->um_gs, 84);
            constexpr int rt = gather_ring_block<84>();
            k_gather_ring<84><<<rgrid, rt, rs, h->stream>>>(pl, h->um_gimg.p, x32p, h->vext32.p, h->w.p, df32, h->partial.p, h->kerr.p, ga, h->um_gs, ntiles);
            red_blocks = rgrid;
        } else if (v84)
            k_gather_umma<84><<<grid, kUmThreads, smem, h->stream>>>(pl, h->um_gimg.p, x32p, h->vext32.p, h->w.p, df32, h->partial.p, h->kerr.p, ga, h->um_gs, ntiles);
        else
            k_gather_umma<0><<<grid, kUmThreads, smem, h->stream>>>(pl, h->um_gimg.p, x32p, h->vext32.p, h->w.p, df32, h->partial.p, h->kerr.p, ga, h->um_gs, ntiles);
        if (!(v84 && h->ring_g)) red_blocks = grid;
    } else if (x32) {
        // FP32 phase of a mixed solve: point, vext, gradient and direction in FP32
        const int ntiles = (int)(g.N / kGtBM);
        const int grid = std::min(ntiles, h->nsm * 2);
        const size_t smem = gather_tma_smem_bytes(g.np, g.no, gt_ncol);
        float *df32 = reinterpret_cast<float *>(d_df);
        const float *x32p = static_cast<const float *>(xin);
        const float2 *pl = (const float2 *)planes;
        const float *B32 = (const float *)B;
        if (gt_ncol == 1)
            k_gather_tma<1><<<grid, kGtThreads, smem, h->stream>>>(pl, B32, x32p, h->vext32.p, h->w.p, df32, h->partial.p, h->kerr.p, ga, ntiles);
        else if (gt_ncol == 2)
            k_gather_tma<2><<<grid, kGtThreads, smem, h->stream>>>(pl, B32, x32p, h->vext32.p, h->w.p, df32, h->partial.p, h->kerr.p, ga, ntiles);
        else
            k_gather_tma<3><<<grid, kGtThreads, smem, h->stream>>>(pl, B32, x32p, h->vext32.p, h->w.p, df32, h->partial.p, h->kerr.p, ga, ntiles);
        red_blocks = grid;
    } else {
        launch_gather_mma<T>(h, planes, d_xi, d_df, ga, vec32);
    }
    if ((rc = check_cuda(cudaGetLastError(), "gather launch"))) return rc;
    h->launches += 3;  // project, oz, gather (the FFT launches are counted in launch_fft_t)
    if (red_blocks) {
        k_reduce_sums<<<1, 256, 0, h->stream>>>(h->partial.p, (int)red_blocks, sums_out(h));
        h->launches += 1;
        if ((rc = check_cuda(cudaGetLastError(), "reduce launch"))) return rc;
    }
    if (has_bridge(h) && do_ideal && (rc = launch_bridge(h, d_xi, ga.df_mode == 1 ? d_df : nullptr, static_cast<const double *>(dvec))))
        return rc;
    stage_mark(h, 5);
    return MDFT_OK;
}

// dvec (df_mode 1 only): h_sums[3] = df.dvec, h_sums[4] = max|df| after finish_sums.
// vec32 (bulk-copy gather only): df and dvec are FP32 vectors (the minimiser's mixed solves);
// x32 (FP32 evaluations, with vec32): the point is FP32 too and vext is read from h->vext32.
// The pipeline is a fixed sequence of launches for given buffers and flags: it runs as a CUDA
// graph captured on first use (one graph launch instead of about a dozen kernel launches per
// evaluation), falling back to direct launches when capture is not possible.
constexpr size_t kMaxPipeGraphs = 8;
void drop_pipe_graphs(mdft_handle *h) {
    for (auto &pg : h->pipe_graphs) cudaGraphExecDestroy(pg.exec);
    h->pipe_graphs.clear();
}
int run_pipeline(mdft_handle *h, const void *d_xi, double *d_df, int do_ideal, int df_mode, const void *dvec = nullptr,
                 bool vec32 = false, bool x32 = false) {
    auto direct = [&]() {
        if (h->eval_prec == MDFT_PREC_MIXED) return run_pipeline_t<float>(h, d_xi, d_df, do_ideal, df_mode, dvec, vec32, x32);
        return run_pipeline_t<double>(h, d_xi, d_df, do_ideal, df_mode, dvec, vec32, x32);
    };
    if (!h->graphs_on || h->timing) return direct();
    for (auto &pg : h->pipe_graphs)
        if (pg.x == d_xi && pg.g == d_df && pg.dvec == dvec && pg.do_ideal == do_ideal && pg.df_mode == df_mode &&
            pg.prec == h->eval_prec && pg.v32 == vec32 && pg.x32 == x32 && pg.vext == h->vext.p && pg.vext32 == h->vext32.p) {
            h->launches += pg.nlaunch;
            return check_cuda(cudaGraphLaunch(pg.exec, h->stream), "pipeline graph launch");
        }
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(h->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return direct();  // inside a caller's capture: launch into it
    }
    const long long l0 = h->launches;
    if (cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return direct();
    }
    const int rc = direct();
    const long long nl = h->launches - l0;  // counted during capture; nothing has run yet
    h->launches = l0;
    cudaGraph_t graph = nullptr;
    const cudaError_t e = cudaStreamEndCapture(h->stream, &graph);
    cudaGraphExec_t exec = nullptr;
    const bool ok = rc == 0 && e == cudaSuccess && graph && cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    if (rc) return rc;  // a launch was refused (nothing ran)
    if (!ok) {
        h->graphs_on = false;  // this handle's pipeline does not capture: launch directly from now on
        return direct();
    }
    if (h->pipe_graphs.size() >= kMaxPipeGraphs) {
        cudaGraphExecDestroy(h->pipe_graphs.front().exec);
        h->pipe_graphs.erase(h->pipe_graphs.begin());
    }
    h->pipe_graphs.push_back(mdft_handle::PipeGraph{d_xi, dvec, h->vext.p, h->vext32.p, d_df, do_ideal, df_mode, h->eval_prec, vec32, x32, exec, nl});
    h->launches += nl;
    return check_cuda(cudaGraphLaunch(exec, h->stream), "pipeline graph launch");
}

// A bridge's error code, once reported: evaluations that run no bridge (the excess term alone)
// do not write it anew.
void clear_bridge_error(mdft_handle *h) {
    cudaMemsetAsync(h->sums.p + 7, 0, sizeof(double), h->stream);
    h->h_sums[7] = 0.0;
}

int finish_sums(mdft_handle *h, double *fid, double *fext, double *fexc) {
    // the pipeline's last kernels left {F_id, F_ext, sum_exc, df.dvec, max|df|, sum w df, F_b,
    // bridge error} and the flag in pinned memory
    int rc;
    if ((rc = check_cuda(cudaStreamSynchronize(h->stream), "evaluation"))) return rc;
    if (*h->h_kerr) {
        cudaMemsetAsync(h->kerr.p, 0, sizeof(int), h->stream);
        set_error("a pipeline wait in the projection or gather timed out (bulk copy never completed)");
        return MDFT_E_CUDA;
    }
    if (h->fmt && h->h_sums[7] != 0.0) {
        const int code = (int)h->h_sums[7];
        clear_bridge_error(h);
        set_error(code == 1 ? "hard-sphere bridge: a weighted density n3 >= 1 (log(1 - n3) undefined)"
                  : code == 2 ? "hard-sphere bridge (CS): a weighted density n3 <= 0"
                              : "hard-sphere bridge: 1 - n3 or n3 at zero in the gradient");
        return MDFT_E_NUMERIC;
    }
    if (h->timing) {
        for (int i = 0; i < ST_COUNT; ++i) {
            float ms = 0;
            cudaEventElapsedTime(&ms, h->ev[i], h->ev[i + 1]);
            h->stage_ms[i] += ms;
        }
        h->stage_count++;
    }
    *fid = h->h_sums[0];
    *fext = h->h_sums[1];
    *fexc = h->h_sums[2] * 0.5 * h->g.dv;
    if (!std::isfinite(*fid) || !std::isfinite(*fext) || !std::isfinite(*fexc)) {
        set_error("non-finite functional (F_id=%g F_ext=%g F_exc=%g)", *fid, *fext, *fexc);
        return MDFT_E_NUMERIC;
    }
    return 0;
}

double combine(const mdft_handle *h, double fid, double fext, double fexc) {
    // src/module_energy_and_gradient.f90:89-217
    double f = 0.0;
    f = f + fid + fext;
    f = f + fexc;
    f = f + (has_bridge(h) ? h->h_sums[6] : 0.0);  // bridge: F_b of this evaluation ("no": 0)
    f = f + h->const_corr;
    return f;
}

// create-time tuning of the FP32 kernel forms (defined with the solver, solve.cuh)
int autotune_at_create(mdft_handle *h);

}  // namespace

// -------------------------------------------------------------------------
extern "C" {

const char *mdft_last_error(void) { return last_error(); }

int mdft_create(const mdft_desc *d, mdft_handle **out) {
    if (!d || !out) { set_error("null argument"); return MDFT_E_ARG; }
    *out = nullptr;
    if (d->nx <= 0 || d->ny <= 0 || d->nz <= 0 || (d->nx & 1) || (d->ny & 1) || (d->nz & 1)) {
        set_error("grid sizes must be positive and even (got %d %d %d)", d->nx, d->ny, d->nz);
        return MDFT_E_ARG;
    }
    if (!(d->lx > 0 && d->ly > 0 && d->lz > 0)) { set_error("box lengths must be positive"); return MDFT_E_ARG; }
    if (d->mmax < 0 || d->mmax > kMaxMmax) { set_error("mmax must be in [0, %d]", kMaxMmax); return MDFT_E_ARG; }
    if (d->mrso < 1) { set_error("mrso must be >= 1"); return MDFT_E_ARG; }
    if (!(d->temperature > 0) || !(d->n0 > 0)) { set_error("temperature and n0 must be positive"); return MDFT_E_ARG; }
    if (d->precision != MDFT_PREC_FP64 && d->precision != MDFT_PREC_MIXED) { set_error("unknown precision %d", d->precision); return MDFT_E_ARG; }
    std::unique_ptr<mdft_handle> h(new mdft_handle());
    {
        const char *tr = std::getenv("MDFT_TRACE");
        h->trace = tr && tr[0] && tr[0] != '0';
        const char *gr = std::getenv("MDFT_GRAPHS");
        h->graphs_on = !(gr && std::strcmp(gr, "0") == 0);
    }
    h->precision = d->precision;
    h->device = d->device;
    // host-side set-up first: argument and c(k) errors do not depend on the device
    const double kT = kBoltz * kNavo * d->temperature * 1.0e-3;  // src/module_thermo.f90:62
    if (build_grid(h->g, d->nx, d->ny, d->nz, d->lx, d->ly, d->lz, d->mmax, d->mrso, kT, d->n0)) return MDFT_E_ARG;
    const Grid &g = h->g;
    if (g.np > kMaxNpConst) { set_error("too many projections (%d)", g.np); return MDFT_E_ARG; }
    {
        FftPlan1D tmp;
        const int dims[3] = {d->nx, d->ny, d->nz};
        for (int ax = 0; ax < 3; ++ax)
            if (!make_plan1d(dims[ax], tmp)) { set_error("grid size %d is not of the form 2^a 3^b", dims[ax]); return MDFT_E_ARG; }
    }
    if (read_ctable(g, d->ck_path, h->ct)) return MDFT_E_IO;
    int rc = check_cuda(cudaSetDevice(d->device), "cudaSetDevice");
    if (rc) return rc;
    if ((rc = check_cuda(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking), "stream"))) return rc;
    for (int i = 0; i <= ST_COUNT; ++i)
        if ((rc = check_cuda(cudaEventCreate(&h->ev[i]), "event"))) return rc;
    const size_t nf = (size_t)g.N * g.no;
    if ((rc = alloc_check(h->xi.alloc(nf), "xi", nf * 8))) return rc;
    if ((rc = alloc_check(h->vext.alloc(nf), "vext", nf * 8))) return rc;
    if ((rc = alloc_check(h->df.alloc(nf), "df", nf * 8))) return rc;
    if ((rc = alloc_check(h->planes.alloc((size_t)g.np * g.N), "projection planes", (size_t)g.np * g.N * 16))) return rc;
    if ((rc = check_cuda(cudaMemsetAsync(h->vext.p, 0, nf * 8, h->stream), "vext clear"))) return rc;
    std::vector<double> A, B;
    build_angular_matrices(g, A, B);
    if ((rc = alloc_check(h->A.alloc(A.size()), "A", A.size() * 8))) return rc;
    if ((rc = alloc_check(h->B.alloc(B.size()), "B", B.size() * 8))) return rc;
    if ((rc = alloc_check(h->w.alloc(g.no), "w", g.no * 8))) return rc;
    cudaMemcpy(h->A.p, A.data(), A.size() * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(h->B.p, B.data(), B.size() * 8, cudaMemcpyHostToDevice);
    {
        std::vector<float> A32(A.begin(), A.end()), B32(B.begin(), B.end());
        if ((rc = alloc_check(h->A32.alloc(A32.size()), "A32", A32.size() * 4))) return rc;
        if ((rc = alloc_check(h->B32.alloc(B32.size()), "B32", B32.size() * 4))) return rc;
        cudaMemcpy(h->A32.p, A32.data(), A32.size() * 4, cudaMemcpyHostToDevice);
        cudaMemcpy(h->B32.p, B32.data(), B32.size() * 4, cudaMemcpyHostToDevice);
        if ((rc = alloc_check(h->planes32.alloc((size_t)g.np * g.N), "FP32 projection planes", (size_t)g.np * g.N * 8))) return rc;
    }
    cudaMemcpy(h->w.p, g.w.data(), g.no * 8, cudaMemcpyHostToDevice);
    if ((rc = alloc_check(h->ctab.alloc((size_t)h->ct.nq * h->ct.ncoef), "c table", h->ct.c.size() * 8))) return rc;
    cudaMemcpy(h->ctab.p, h->ct.c.data(), h->ct.c.size() * 8, cudaMemcpyHostToDevice);
    {
        std::vector<float> c32(h->ct.c.begin(), h->ct.c.end());
        if ((rc = alloc_check(h->ctab32.alloc((size_t)h->ct.nq * h->ct.ncoef), "FP32 c table", c32.size() * 4))) return rc;
        cudaMemcpy(h->ctab32.p, c32.data(), c32.size() * 4, cudaMemcpyHostToDevice);
    }
    if ((rc = check_cuda(cudaGetLastError(), "table upload"))) return rc;
    // launch shapes
    int maxsmem = 0;
    cudaDeviceGetAttribute(&maxsmem, cudaDevAttrMaxSharedMemoryPerBlockOptin, d->device);
    const size_t dyn_max = (size_t)maxsmem - 1024;  // static shared memory of these kernels is < 1 KB
    for (const void *fn : {(const void *)k_fft_axis<double>, (const void *)k_fft_axis<float>})
        if ((rc = allow_smem(fn, maxsmem))) return rc;
    for (int n : {g.nx, g.ny, g.nz})
        if ((rc = setup_fft_smem<double>(n, maxsmem)) || (rc = setup_fft_smem<float>(n, maxsmem))) return rc;
    cudaDeviceGetAttribute(&h->nsm, cudaDevAttrMultiProcessorCount, d->device);
    {
        // persistent bulk-copy gather: N a multiple of 32 (two of its tiles), no <= 96, stages that fit
        const int ncol = (g.no + 31) / 32;
        const bool shape_ok = g.N % (2 * kGtBM) == 0 && ncol <= 3;
        h->gt_ncol32 = (shape_ok && gather_tma_smem_bytes(g.np, g.no, ncol) <= dyn_max) ? ncol : 0;
        // persistent bulk-copy projection: N in whole 64-point tiles, np <= 32
        const bool pshape = g.N % kPtBM == 0 && g.np <= 32;
        h->pt_ok32 = pshape && project_tma_smem_bytes(g.np, g.no) <= dyn_max;
        if ((rc = allow_smem((const void *)k_project_tma, maxsmem))) return rc;
        {
            int b = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_project_tma, 256,
                                                          project_tma_smem_bytes(g.np, g.no));
            h->pt_grid_x32 = h->nsm * std::max(1, b);
        }
        for (const void *fn : {(const void *)k_gather_tma<1>, (const void *)k_gather_tma<2>, (const void *)k_gather_tma<3>})
            if ((rc = allow_smem(fn, maxsmem))) return rc;
    }
    {
        double2 lt[kLogN];
        dm_log_table(lt);
        if ((rc = alloc_check(h->dm_log.alloc(kLogN), "logarithm table", sizeof lt))) return rc;
        cudaMemcpy(h->dm_log.p, lt, sizeof lt, cudaMemcpyHostToDevice);
        if ((rc = setup_mma<double>(h.get(), A, B, dyn_max, maxsmem))) return rc;
    }
    {
        // tensor-core angular contractions for FP32 evaluations: N in whole 128-point tiles,
        // no <= 96, 2np <= 64 (mmax <= 3 for water); MDFT_ANGULAR=ffma keeps the FFMA kernels
        const char *ang = std::getenv("MDFT_ANGULAR");
        const bool want = !(ang && std::strcmp(ang, "ffma") == 0);
        // "umma": register forms only; "ring": the bulk-copy ring forms of both contractions;
        // default: register projection (measured faster) and ring gather
        const bool want_ring = !(ang && std::strcmp(ang, "umma") == 0);
        const bool want_ring_p = ang && std::strcmp(ang, "ring") == 0;
        h->um_ps = umma_shape(g.no, 2 * g.np);
        h->um_gs = umma_shape(2 * g.np, g.no);
        if (want && g.N % kUmBM == 0 && h->um_ps.Kp <= 96 && h->um_gs.Kp <= 64 &&
            gather_umma_smem_bytes(h->um_gs, g.no) <= dyn_max && umma_smem_bytes(h->um_ps) <= dyn_max) {
            std::vector<uint16_t> pimg, gimg;
            const int np2 = 2 * g.np, no = g.no;
            pack_split_bf16(h->um_ps.Np, h->um_ps.Kp, [&](int n, int io) { return (n < np2 && io < no) ? A[(size_t)io * np2 + n] : 0.0; }, pimg);
            pack_split_bf16(h->um_gs.Np, h->um_gs.Kp, [&](int io, int k) { return (io < no && k < np2) ? B[(size_t)k * no + io] : 0.0; }, gimg);
            if ((rc = alloc_check(h->um_pimg.alloc(pimg.size()), "angular operand images", pimg.size() * 2))) return rc;
            if ((rc = alloc_check(h->um_gimg.alloc(gimg.size()), "angular operand images", gimg.size() * 2))) return rc;
            cudaMemcpy(h->um_pimg.p, pimg.data(), pimg.size() * 2, cudaMemcpyHostToDevice);
            cudaMemcpy(h->um_gimg.p, gimg.data(), gimg.size() * 2, cudaMemcpyHostToDevice);
            const void *pf[] = {(const void *)k_project_umma<4>, (const void *)k_project_umma<1>};
            const void *gf[] = {(const void *)k_gather_umma<84>, (const void *)k_gather_umma<0>};
            for (const void *fn : pf)
                if ((rc = allow_smem(fn, maxsmem))) return rc;
            for (const void *fn : gf)
                if ((rc = allow_smem(fn, maxsmem))) return rc;
            int bp = 0, bg = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bp, k_project_umma<4>, kPjThreads, umma_smem_bytes(h->um_ps));
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bg, k_gather_umma<84>, kUmThreads,
                                                          gather_umma_smem_bytes(h->um_gs, g.no));
            h->um_grid_p = h->nsm * std::max(1, bp);
            h->um_grid_g = h->nsm * std::max(1, bg);
            h->um_ok = true;
            h->ring_p_ok = project_ring_smem_bytes(h->um_ps, g.no) <= dyn_max;
            h->ring_g_ok = g.no == 84 && gather_ring_smem_bytes(h->um_gs, 84) <= dyn_max;
            h->ring_p = want_ring_p && h->ring_p_ok;
            h->ring_g = want_ring && h->ring_g_ok;
            if (h->ring_p_ok) {
                if ((rc = allow_smem((const void *)k_project_ring<4>, maxsmem))) return rc;
                if ((rc = allow_smem((const void *)k_project_ring<1>, maxsmem))) return rc;
            }
            if (h->ring_g_ok && (rc = allow_smem((const void *)k_gather_ring<84>, maxsmem))) return rc;
            // the FP32 forms are measured on the first FP32 phase unless chosen in the environment
            const char *at = std::getenv("MDFT_AUTOTUNE");
            h->tune_on = !(at && std::strcmp(at, "0") == 0) && !ang && !std::getenv("MDFT_OZ");
        }
    }
    {
        // k_gather_mma's grids: at most what an SM's threads hold
        const size_t rows = std::max<long long>({2LL * h->nsm, (long long)h->um_grid_g, (long long)h->dm_g[0].grid, (long long)(2048 / kGmThreads) * h->nsm});
        if ((rc = alloc_check(h->partial.alloc(kGatherSums * rows), "partials", 8 * kGatherSums * rows))) return rc;
    }
    if ((rc = alloc_check(h->kerr.alloc(2), "error flag", 8))) return rc;
    cudaMemset(h->kerr.p, 0, 2 * sizeof(int));
    if ((rc = check_cuda(cudaMallocHost(&h->h_kerr, sizeof(int)), "pinned flag"))) return rc;
    *h->h_kerr = 0;
    if ((rc = alloc_check(h->sums.alloc(8), "sums", 64))) return rc;
    cudaMemset(h->sums.p, 0, 8 * sizeof(double));
    if ((rc = check_cuda(cudaMallocHost(&h->h_sums, 8 * sizeof(double)), "pinned sums"))) return rc;
    std::fill(h->h_sums, h->h_sums + 8, 0.0);
    if ((rc = alloc_check(h->vpart.alloc((size_t)kMaxRows * kRedBlocks), "reduction partials", 8 * kMaxRows * kRedBlocks))) return rc;
    if ((rc = alloc_check(h->vsc.alloc(kScalarSlots), "reduction scalars", 8 * kScalarSlots))) return rc;
    if ((rc = check_cuda(cudaMallocHost(&h->h_vsc, sizeof(double) * kScalarSlots), "pinned scalars"))) return rc;
    if ((rc = setup_fft(h.get()))) return rc;
    for (int ax = 0; ax < 3; ++ax)
        if (h->fft[ax].smem > (size_t)maxsmem) { set_error("FFT tile does not fit in shared memory"); return MDFT_E_ARG; }
    {
        OzTables tb;
        if (!build_oz_tables(g, h->ct, tb)) { set_error("OZ term tables exceed their index encoding"); return MDFT_E_ARG; }
        if ((rc = alloc_check(h->oz_ints.alloc(tb.ints.size()), "OZ tables", tb.ints.size() * 4))) return rc;
        if ((rc = alloc_check(h->oz_dbls.alloc(std::max<size_t>(1, tb.dbls.size())), "OZ tables", tb.dbls.size() * 8))) return rc;
        cudaMemcpy(h->oz_ints.p, tb.ints.data(), tb.ints.size() * 4, cudaMemcpyHostToDevice);
        if (!tb.dbls.empty()) cudaMemcpy(h->oz_dbls.p, tb.dbls.data(), tb.dbls.size() * 8, cudaMemcpyHostToDevice);
        Oz2Args &oz = h->oz;
        oz.nx = g.nx; oz.ny = g.ny; oz.nz = g.nz; oz.N = g.N;
        oz.nk = (long long)g.nx * g.ny * (g.nz / 2 + 1);
        oz.mmax = g.mmax; oz.np = g.np; oz.ncoef = h->ct.ncoef; oz.nq = h->ct.nq; oz.dq = h->ct.dq;
        oz.twopi_lx = 2.0 * kPi / g.lx; oz.twopi_ly = 2.0 * kPi / g.ly; oz.twopi_lz = 2.0 * kPi / g.lz;
        oz.quirks = 1;
        oz.n_ints = (int)tb.ints.size(); oz.n_dbls = (int)tb.dbls.size(); oz.nrot = tb.nrot;
        oz.fwd_off = tb.fwd_off; oz.fwd_terms = tb.fwd_terms; oz.oz_off = tb.oz_off; oz.oz_terms = tb.oz_terms;
        oz.bwd_off = tb.bwd_off; oz.bwd_terms = tb.bwd_terms; oz.sign = tb.sign; oz.lvl_off = tb.lvl_off;
        oz.rec_int = tb.rec_int;
        if (g.mrso == 2 || g.mmax == 0) {
            OzcArgs &a = h->ozc;
            a.nx = g.nx; a.ny = g.ny; a.nz = g.nz;
            a.hx = g.nx / 2 + 1; a.hy = g.ny / 2 + 1;
            a.N = g.N;
            a.ncell = a.hx * a.hy * (g.nz / 2 + 1);
            std::vector<int> xu;
            std::vector<double> cf;
            build_ozc_recipes(g.mmax, xu, cf);
            if (!xu.empty()) {
                if ((rc = alloc_check(h->ozc_xu.alloc(xu.size()), "OZ recursion", xu.size() * 4))) return rc;
                if ((rc = alloc_check(h->ozc_cf.alloc(cf.size()), "OZ recursion", cf.size() * 8))) return rc;
                cudaMemcpy(h->ozc_xu.p, xu.data(), xu.size() * 4, cudaMemcpyHostToDevice);
                cudaMemcpy(h->ozc_cf.p, cf.data(), cf.size() * 8, cudaMemcpyHostToDevice);
            }
            const std::vector<double> cx = build_ozc_table(g, h->ct);
            if ((rc = setup_ozc<double>(h.get(), cx, h->ozc_c64, h->ozc_rec64, h->ozc_grid64, maxsmem))) return rc;
            h->ozc_ok = true;
        } else {
            auto shape = [&](auto tag, const void *fn, int i) {
                using T = decltype(tag);
                int &W = h->oz_warps[i];
                W = 8;
                while (W > 1 && oz2_smem_bytes<T>(oz, W) > dyn_max) W /= 2;
                h->oz_smem[i] = oz2_smem_bytes<T>(oz, W);
                if (h->oz_smem[i] > dyn_max) { set_error("OZ tile does not fit in shared memory"); return (int)MDFT_E_ARG; }
                const int r = allow_smem(fn, maxsmem);
                if (r) return r;
                // persistent grid: as many CTAs as fit on the device at once (tables staged once per CTA)
                int per_sm = 0;
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 32 * W, h->oz_smem[i]);
                h->oz_grid[i] = (int)std::min<long long>((oz.nk + W - 1) / W, (long long)std::max(1, per_sm) * h->nsm);
                return 0;
            };
            if ((rc = shape(0.0, (const void *)k_oz2<double>, 0)) || (rc = shape(0.f, (const void *)k_oz2<float>, 1))) return rc;
        }
        // thread-per-pair FP32 OZ where an instantiation exists and its slice fits
        const void *fn = ozp_kernel(g.mmax, g.mrso);
        if (fn && build_ozp_params(g, h->ct, h->ozp) && ozp_smem_bytes(g.np) <= dyn_max) {
            if ((rc = allow_smem(fn, maxsmem))) return rc;
            h->ozp_ok = true;
            const char *ozsel = std::getenv("MDFT_OZ");
            h->ozd = !(ozsel && std::strcmp(ozsel, "ozp") == 0);
        }
    }
    h->eval_prec = h->precision;
    if (h->precision == MDFT_PREC_MIXED && (rc = ensure_fp32(h.get()))) return rc;
    if ((rc = autotune_at_create(h.get()))) return rc;
    if ((rc = check_cuda(cudaStreamSynchronize(h->stream), "create"))) return rc;
    *out = h.release();
    return MDFT_OK;
}

int mdft_destroy(mdft_handle *h) {
    if (!h) return MDFT_OK;
    if (h->stream) cudaStreamSynchronize(h->stream);
    // an attached warm-start network goes back to its own stream before this one is destroyed
    if (h->warm) mdft_warm_net_set_stream(h->warm, nullptr);
    h->warm = nullptr;
    drop_pipe_graphs(h);
    h->ozp_cq.free();
    h->um_pimg.free();
    h->um_gimg.free();
    h->xi.free(); h->vext.free(); h->vext32.free(); h->df.free(); h->w.free(); h->A.free(); h->B.free();
    h->partial.free(); h->sums.free(); h->planes.free(); h->ctab.free(); h->oz_ints.free(); h->oz_dbls.free();
    for (int i = 0; i < 3; ++i) {
        h->tw64[i].free();
        h->tw32[i].free();
    }
    h->A32.free(); h->B32.free(); h->planes32.free(); h->ctab32.free();
    lbfgs_free(h->lb);
    h->vpart.free();
    h->vsc.free();
    if (h->h_vsc) cudaFreeHost(h->h_vsc);
    if (h->h_sums) cudaFreeHost(h->h_sums);
    if (h->h_kerr) cudaFreeHost(h->h_kerr);
    h->kerr.free();
    for (int i = 0; i <= ST_COUNT; ++i)
        if (h->ev[i]) cudaEventDestroy(h->ev[i]);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return MDFT_OK;
}

int mdft_get_sizes(const mdft_handle *h, mdft_sizes *o) {
    if (!h || !o) { set_error("null argument"); return MDFT_E_ARG; }
    o->ntheta = h->g.ntheta; o->nphi = h->g.nphi; o->npsi = h->g.npsi;
    o->no = h->g.no; o->np = h->g.np;
    o->ncoef = h->ct.ncoef; o->nq = h->ct.nq;
    o->dv = h->g.dv; o->rho0 = h->g.rho0; o->kT = h->g.kT; o->dq = h->ct.dq;
    return MDFT_OK;
}

int mdft_get_stream(const mdft_handle *h, void **s) {
    if (!h || !s) { set_error("null argument"); return MDFT_E_ARG; }
    *s = (void *)h->stream;
    return MDFT_OK;
}

int mdft_get_weights(const mdft_handle *h, double *w) {
    if (!h || !w) { set_error("null argument"); return MDFT_E_ARG; }
    std::memcpy(w, h->g.w.data(), sizeof(double) * h->g.no);
    return MDFT_OK;
}

int mdft_set_vext(mdft_handle *h, const double *v) {
    if (!h || !v) { set_error("null argument"); return MDFT_E_ARG; }
    size_t n = (size_t)h->g.N * h->g.no;
    int rc = check_cuda(cudaMemcpyAsync(h->vext.p, v, n * 8, cudaMemcpyHostToDevice, h->stream), "vext upload");
    if (rc) return rc;
    if ((rc = check_cuda(cudaStreamSynchronize(h->stream), "vext upload"))) return rc;
    h->have_vext = true;
    return MDFT_OK;
}

int mdft_get_vext(const mdft_handle *h, double *v) {
    if (!h || !v) { set_error("null argument"); return MDFT_E_ARG; }
    size_t n = (size_t)h->g.N * h->g.no;
    int rc = check_cuda(cudaMemcpyAsync(v, h->vext.p, n * 8, cudaMemcpyDeviceToHost, h->stream), "vext download");
    if (rc) return rc;
    return check_cuda(cudaStreamSynchronize(h->stream), "vext download");
}

int mdft_set_constant_correction(mdft_handle *h, double c) {
    if (!h) { set_error("null argument"); return MDFT_E_ARG; }
    h->const_corr = c;
    return MDFT_OK;
}

// c00_000 by solvent(1)%name and grid%mmax (src/module_coarse_grained_gageat_bridge.f90:260-263)
int mdft_cgb_c00(const char *solvent, int mmax, double *c00) {
    if (!solvent || !c00) { set_error("null argument"); return MDFT_E_ARG; }
    if (std::strcmp(solvent, "spce") == 0) *c00 = mmax == 0 ? -14.64872 : -13.665;
    else if (std::strcmp(solvent, "tip3p") == 0) *c00 = -11.9078;
    else {
        set_error("no c00_000 for solvent '%s' (the reference has values for spce and tip3p only)", solvent);
        return MDFT_E_ARG;
    }
    return MDFT_OK;
}

}  // extern "C"

namespace {
// bridge = "no": drop both terms and their buffers
int clear_bridges(mdft_handle *h) {
    drop_pipe_graphs(h);  // the captured pipelines carry the bridge's launches
    h->cgb = 0;
    h->fmt = 0;
    h->cgb_kk.free(); h->cgb_a.free(); h->cgb_b.free(); h->cgb_dens.free(); h->cgb_part.free();
    h->fmt_pl.free(); h->fmt_cs.free(); h->fmt_part.free();
    h->h_sums[6] = h->h_sums[7] = 0.0;
    return check_cuda(cudaMemsetAsync(h->sums.p + 6, 0, 2 * sizeof(double), h->stream), "sums reset");
}
}  // namespace

extern "C" {

int mdft_set_bridge_cgb(mdft_handle *h, int version, double B6, double sigma, double c00) {
    if (!h) { set_error("null argument"); return MDFT_E_ARG; }
    if (version < MDFT_BRIDGE_NONE || version > MDFT_BRIDGE_CGB_WDA) { set_error("unknown cgb version %d", version); return MDFT_E_ARG; }
    if (version != MDFT_BRIDGE_NONE && h->precision != MDFT_PREC_FP64) {
        set_error("the bridge term needs an FP64 handle");
        return MDFT_E_ARG;
    }
    if (version != MDFT_BRIDGE_NONE && !(sigma > 0.0 && std::isfinite(sigma) && std::isfinite(B6) && std::isfinite(c00))) {
        set_error("cgb parameters must be finite, sigma > 0");
        return MDFT_E_ARG;
    }
    int rc = clear_bridges(h);
    if (rc || version == MDFT_BRIDGE_NONE) return rc;
    const Grid &g = h->g;
    if ((rc = alloc_check(h->cgb_kk.alloc(g.N), "bridge kernel", g.N * 16))) return rc;
    if ((rc = alloc_check(h->cgb_a.alloc(g.N), "bridge plane", g.N * 16))) return rc;
    if ((rc = alloc_check(h->cgb_b.alloc(g.N), "bridge plane", g.N * 16))) return rc;
    if ((rc = alloc_check(h->cgb_dens.alloc(g.N), "bridge density", g.N * 8))) return rc;
    if ((rc = alloc_check(h->cgb_part.alloc(4 * kRedBlocks), "bridge partials", 32 * kRedBlocks))) return rc;
    // fill_kernel (src/module_coarse_grained_gageat_bridge.f90:123-210)
    const double pi = std::acos(-1.0);
    const double sp = sigma * std::sqrt(2.0 * pi);
    const double gp = 1.0 / (sp * sp * sp), oo = 1.0 / (2.0 * sigma * sigma);
    const double cut = -1.0 / oo * std::log(1.0e-10 / gp);
    const double nf = (double)(float)(g.nx * g.ny * g.nz);  // real(nx*ny*nz): single precision
    k_cgb_kernel<<<kRedBlocks, kBrThreads, 0, h->stream>>>(h->cgb_kk.p, g.nx, g.ny, g.nz, g.lx / g.nx, g.ly / g.ny, g.lz / g.nz,
                                                           gp, oo, cut);
    if ((rc = launch_fft_planes(h, h->cgb_kk.p, 1, -1))) return rc;
    k_cgb_scale<<<kRedBlocks, kBrThreads, 0, h->stream>>>(h->cgb_kk.p, g.N, nf, g.lx * g.ly * g.lz);
    h->launches += 2;
    if ((rc = check_cuda(cudaGetLastError(), "bridge kernel"))) return rc;
    CgbArgs &a = h->cgb_args;
    a.N = g.N;
    a.no = g.no;
    a.version = version;
    a.rho0 = g.rho0;
    a.n0 = g.n0;
    a.kT = g.kT;
    a.vvox = (g.lx / g.nx) * (g.ly / g.ny) * (g.lz / g.nz);
    a.nf = nf;
    a.A3 = 1.0 - c00 / 2.0;
    a.B6 = B6;
    h->cgb = version;
    return check_cuda(cudaStreamSynchronize(h->stream), "bridge set-up");
}

// The bulk hard-sphere parameters (src/module_hardspheres.f90:83-189) and the hard-sphere
// c(k) (src/cs_of_k_hard_sphere.f90:56-157) on nb_k points of the c(k) file's step.
int mdft_set_bridge_fmt(mdft_handle *h, int functional, double R) {
    if (!h) { set_error("null argument"); return MDFT_E_ARG; }
    if (functional < MDFT_BRIDGE_NONE || functional > MDFT_BRIDGE_HS_CS) { set_error("unknown hard-sphere functional %d", functional); return MDFT_E_ARG; }
    if (functional != MDFT_BRIDGE_NONE && h->precision != MDFT_PREC_FP64) {
        set_error("the bridge term needs an FP64 handle");
        return MDFT_E_ARG;
    }
    if (functional != MDFT_BRIDGE_NONE && !(R > 0.0 && std::isfinite(R))) { set_error("the hard-sphere radius must be positive"); return MDFT_E_ARG; }
    int rc = clear_bridges(h);
    if (rc || functional == MDFT_BRIDGE_NONE) return rc;
    const Grid &g = h->g;
    const double pi = kPi, kT = g.kT, n0 = g.n0;
    const double pf = (double)(4.0f / 3.0f) * pi * n0 * (R * R * R);  // fourthird = 4./3. (single)
    if (pf >= 0.74) { set_error("hard-sphere packing fraction %g is above 0.74", pf); return MDFT_E_ARG; }
    // excess chemical potential and bulk grand potential
    const double b1 = n0 * R, b2 = n0 * 4 * pi * (R * R), b3 = n0 * 4 * pi * (R * R * R) / 3;
    double dp[4];
    dp[0] = -std::log(1 - b3);
    dp[1] = b2 / (1 - b3);
    if (functional == MDFT_BRIDGE_HS_PY) {
        dp[2] = b1 / (1 - b3) + (b2 * b2) / (8 * pi * ((1 - b3) * (1 - b3)));
        dp[3] = n0 / (1 - b3) + b1 * b2 / ((1 - b3) * (1 - b3)) + (b2 * b2 * b2) / (12 * pi * ((1 - b3) * (1 - b3) * (1 - b3)));
    } else {
        const double m = b3 - 1;
        dp[2] = (b3 * ((b2 * b2) - 12 * b1 * m * b3 * pi) + (b2 * b2) * (m * m) * std::log(1 - b3)) / (12 * pi * (m * m) * (b3 * b3));
        dp[3] = (b3 * ((b2 * b2 * b2) * (2 - 5 * b3 + (b3 * b3)) + 36 * b1 * b2 * m * (b3 * b3) * pi - 36 * n0 * (m * m) * (b3 * b3) * pi) -
                 2 * (b2 * b2 * b2) * (m * m * m) * std::log(1 - b3)) /
                (36 * pi * (m * m * m) * (b3 * b3 * b3));
    }
    const double dn[4] = {1, R, 4 * pi * (R * R), 4 * pi * (R * R * R) / 3.0};
    double acc = 0.0;
    for (int i = 0; i < 4; ++i) acc += dp[i] * dn[i];
    const double mu = kT * acc;
    double f0 = functional == MDFT_BRIDGE_HS_PY
                    ? kT * (-n0 * std::log(1 - b3) + b1 * b2 / (1 - b3) + (b2 * b2 * b2) / (24 * pi * ((1 - b3) * (1 - b3))))
                    : kT * (((1.0 / (36 * pi)) * (b2 * b2 * b2) / (b3 * b3) - n0) * std::log(1 - b3) + b1 * b2 / (1 - b3) +
                            (1.0 / (36 * pi)) * (b2 * b2 * b2) / (((1 - b3) * (1 - b3)) * b3));
    f0 = (f0 - mu * n0) * (g.lx * g.ly * g.lz);
    // c_hs(k) at k = (i-1) dq with the bulk weighted densities
    const double twopi = 2.0 * pi;
    const double kxm = (double)(g.nx / 2) * twopi / g.lx, kym = (double)(g.ny / 2) * twopi / g.ly, kzm = (double)(g.nz / 2) * twopi / g.lz;
    const double dq = h->ct.dq;
    const int nbk = (int)(std::sqrt(kxm * kxm + kym * kym + kzm * kzm) / dq) + 1;
    std::vector<double> cs(nbk);
    // the bulk weighted densities as cs_of_k_hard_sphere forms them: n0 times w_a(k = 0)
    const double c0 = n0 * 1.0, c1 = n0 * R, c2 = n0 * (4.0 * pi * (R * R)), c3 = n0 * (4.0 * pi / 3.0 * (R * R * R));
    const double u = 1.0 - c3, m1 = -1.0 + c3;
    if (std::fabs(c3 - 1) <= kEpsDp) { set_error("n3 = 1 in the hard-sphere c(k)"); return MDFT_E_ARG; }
    double d[4][4] = {{0}};
    if (functional == MDFT_BRIDGE_HS_PY) {
        d[0][3] = 1.0 / u;
        d[1][2] = 1.0 / u;
        d[1][3] = c2 / (u * u);
        d[2][2] = c2 / (4 * pi * (u * u));
        d[2][3] = c1 / (u * u) + (c2 * c2) / (4 * pi * (u * u * u));
        d[3][3] = (2.0 * c1 * c2) / (u * u * u) + c0 / (u * u) + (c2 * c2 * c2) / (4.0 * pi * ((u * u) * (u * u)));
    } else {
        d[0][3] = 1.0 / (1 - c3);
        d[1][2] = 1.0 / (1.0 - c3);
        d[1][3] = c2 / ((1.0 - c3) * (1.0 - c3));
        d[2][2] = c2 / (6.0 * ((1.0 - c3) * (1.0 - c3)) * c3 * pi) + (c2 * std::log(1.0 - c3)) / (6.0 * (c3 * c3) * pi);
        d[2][3] = (c3 * ((c2 * c2) * (2.0 - 5.0 * c3 + (c3 * c3)) + 12.0 * c1 * m1 * (c3 * c3) * pi) -
                   2.0 * (c2 * c2) * (m1 * m1 * m1) * std::log(1 - c3)) /
                  (12.0 * (m1 * m1 * m1) * (c3 * c3 * c3) * pi);
        d[3][3] = (c3 * ((c2 * c2 * c2) * (6.0 - 21.0 * c3 + 26.0 * (c3 * c3) - 5.0 * (c3 * c3 * c3)) -
                         72.0 * c1 * c2 * m1 * (c3 * c3 * c3) * pi + 36.0 * c0 * (m1 * m1) * (c3 * c3 * c3) * pi) +
                   6.0 * (c2 * c2 * c2) * ((m1 * m1) * (m1 * m1)) * std::log(1.0 - c3)) /
                  (36.0 * ((m1 * m1) * (m1 * m1)) * ((c3 * c3) * (c3 * c3)) * pi);
    }
    d[2][1] = d[1][2];
    d[3][0] = d[0][3];
    d[3][1] = d[1][3];
    d[3][2] = d[2][3];
    for (int i = 0; i < nbk; ++i) {
        const double k = i * dq;
        double w[4];
        if (std::fabs(k) <= kEpsDp) {
            w[0] = 1.0; w[1] = R; w[2] = 4.0 * pi * (R * R); w[3] = 4.0 * pi / 3.0 * (R * R * R);
        } else {
            const double kR = k * R, sk = std::sin(kR), ck = std::cos(kR);
            w[0] = ck + kR * sk / 2.0;
            w[1] = (sk + kR * ck) / (2.0 * k);
            w[2] = (4.0 * pi * R * sk) / k;
            w[3] = 4.0 * pi * (sk - kR * ck) / (k * k * k);
        }
        double sum = 0.0;
        for (int a = 0; a < 4; ++a)
            for (int b = 0; b < 4; ++b) sum += d[a][b] * w[a] * w[b];
        cs[i] = -sum;
    }
    const size_t nb = kRedBlocks;
    if ((rc = alloc_check(h->fmt_pl.alloc(7 * (size_t)g.N), "bridge planes", 7 * 16 * (size_t)g.N))) return rc;
    if ((rc = alloc_check(h->fmt_cs.alloc(nbk), "hard-sphere c(k)", 8 * (size_t)nbk))) return rc;
    if ((rc = alloc_check(h->fmt_part.alloc(10 * nb + 2), "bridge partials", 8 * (10 * nb + 2)))) return rc;
    if ((rc = check_cuda(cudaMemcpy(h->fmt_cs.p, cs.data(), 8 * (size_t)nbk, cudaMemcpyHostToDevice), "hard-sphere c(k)"))) return rc;
    FmtArgs &a = h->fmt_args;
    a.N = g.N;
    a.no = g.no;
    a.nx = g.nx;
    a.ny = g.ny;
    a.nz = g.nz;
    a.version = functional;
    a.rho0 = g.rho0;
    a.kT = kT;
    a.dv = g.dv;
    a.R = R;
    a.mu = mu;
    a.fexc0 = f0;
    a.shift = (twopi * (4.0 * pi)) / (double)g.mrso;
    a.nd = (double)(g.nx * g.ny * g.nz);
    a.dq = dq;
    a.lx = g.lx;
    a.ly = g.ly;
    a.lz = g.lz;
    a.nbk = nbk;
    h->fmt = functional;
    return MDFT_OK;
}

int mdft_get_bridge_fmt_params(const mdft_handle *h, double *out) {
    if (!h || !out) { set_error("null argument"); return MDFT_E_ARG; }
    if (!h->fmt) { set_error("no hard-sphere bridge set"); return MDFT_E_STATE; }
    out[0] = h->fmt_args.R;
    out[1] = h->fmt_args.mu;
    out[2] = h->fmt_args.fexc0;
    out[3] = h->fmt_args.nbk;
    return MDFT_OK;
}

int mdft_bridge_energy(mdft_handle *h, const double *xi, double *fb, double *df) {
    if (!h || !xi || !fb) { set_error("null argument"); return MDFT_E_ARG; }
    *fb = 0.0;
    if (!has_bridge(h)) return MDFT_OK;  // bridge "no"
    const size_t n = (size_t)h->g.N * h->g.no;
    int rc = check_cuda(cudaMemcpyAsync(h->xi.p, xi, n * 8, cudaMemcpyHostToDevice, h->stream), "xi upload");
    if (rc) return rc;
    if (df && (rc = check_cuda(cudaMemcpyAsync(h->df.p, df, n * 8, cudaMemcpyHostToDevice, h->stream), "df upload"))) return rc;
    if ((rc = launch_bridge(h, h->xi.p, df ? h->df.p : nullptr, nullptr))) return rc;
    if ((rc = check_cuda(cudaMemcpyAsync(h->h_sums + 6, h->sums.p + 6, 2 * sizeof(double), cudaMemcpyDeviceToHost, h->stream), "sums copy")))
        return rc;
    if (df && (rc = check_cuda(cudaMemcpyAsync(df, h->df.p, n * 8, cudaMemcpyDeviceToHost, h->stream), "df download"))) return rc;
    if ((rc = check_cuda(cudaStreamSynchronize(h->stream), "bridge"))) return rc;
    if (h->fmt && h->h_sums[7] != 0.0) {
        set_error("hard-sphere bridge: a weighted density left (0, 1) (code %d)", (int)h->h_sums[7]);
        clear_bridge_error(h);
        return MDFT_E_NUMERIC;
    }
    *fb = h->h_sums[6];
    if (!std::isfinite(*fb)) { set_error("non-finite bridge energy"); return MDFT_E_NUMERIC; }
    return MDFT_OK;
}

int mdft_energy_and_gradient_device(mdft_handle *h, const double *d_xi, double *d_df, double *f, double *terms) {
    if (!h || !d_xi || !f) { set_error("null argument"); return MDFT_E_ARG; }
    int rc = run_pipeline(h, d_xi, d_df, 1, 1);
    if (rc) return rc;
    double fid, fext, fexc;
    if ((rc = finish_sums(h, &fid, &fext, &fexc))) return rc;
    *f = combine(h, fid, fext, fexc);
    if (terms) {
        terms[0] = fid;
        terms[1] = fext;
        terms[2] = fexc;
        terms[3] = h->const_corr;
    }
    return MDFT_OK;
}

int mdft_energy_and_gradient(mdft_handle *h, const double *xi, double *f, double *df, double *terms) {
    if (!h || !xi || !f) { set_error("null argument"); return MDFT_E_ARG; }
    size_t n = (size_t)h->g.N * h->g.no;
    int rc = check_cuda(cudaMemcpyAsync(h->xi.p, xi, n * 8, cudaMemcpyHostToDevice, h->stream), "xi upload");
    if (rc) return rc;
    if ((rc = mdft_energy_and_gradient_device(h, h->xi.p, df ? h->df.p : nullptr, f, terms))) return rc;
    if (df) {
        if ((rc = check_cuda(cudaMemcpyAsync(df, h->df.p, n * 8, cudaMemcpyDeviceToHost, h->stream), "df download"))) return rc;
        if ((rc = check_cuda(cudaStreamSynchronize(h->stream), "df download"))) return rc;
    }
    return MDFT_OK;
}

int mdft_excess_energy(mdft_handle *h, const double *xi, double *fexc, double *df) {
    if (!h || !xi || !fexc) { set_error("null argument"); return MDFT_E_ARG; }
    size_t n = (size_t)h->g.N * h->g.no;
    int rc = check_cuda(cudaMemcpyAsync(h->xi.p, xi, n * 8, cudaMemcpyHostToDevice, h->stream), "xi upload");
    if (rc) return rc;
    if (df && (rc = check_cuda(cudaMemcpyAsync(h->df.p, df, n * 8, cudaMemcpyHostToDevice, h->stream), "df upload"))) return rc;
    if ((rc = run_pipeline(h, h->xi.p, df ? h->df.p : nullptr, 0, 2))) return rc;
    double a, b;
    if ((rc = finish_sums(h, &a, &b, fexc))) return rc;
    if (df) {
        if ((rc = check_cuda(cudaMemcpyAsync(df, h->df.p, n * 8, cudaMemcpyDeviceToHost, h->stream), "df download"))) return rc;
        if ((rc = check_cuda(cudaStreamSynchronize(h->stream), "df download"))) return rc;
    }
    return MDFT_OK;
}

int mdft_set_timing(mdft_handle *h, int on) {
    if (!h) { set_error("null argument"); return MDFT_E_ARG; }
    h->timing = on != 0;
    for (int i = 0; i < ST_COUNT; ++i) h->stage_ms[i] = 0;
    h->stage_count = 0;
    return MDFT_OK;
}

int mdft_set_wait_failure(mdft_handle *h, int on) {
    if (!h) { set_error("null argument"); return MDFT_E_ARG; }
    h->wait_fail = on != 0;
    drop_pipe_graphs(h);  // the captured launches carry the flag
    return MDFT_OK;
}

int mdft_get_kernel_forms(const mdft_handle *h, int *forms, double *ms) {
    if (!h || !forms) { set_error("null argument"); return MDFT_E_ARG; }
    forms[0] = h->ring_p ? 1 : 0;
    forms[1] = h->ring_g ? 1 : 0;
    forms[2] = h->ozd;
    forms[3] = h->tuned && h->tune_ms[0][0] >= 0 ? 1 : 0;
    if (ms)
        for (int i = 0; i < 3; ++i)
            for (int c = 0; c < 2; ++c) ms[2 * i + c] = h->tune_ms[i][c];
    return MDFT_OK;
}

int mdft_get_launch_count(const mdft_handle *h, long long *count) {
    if (!h || !count) { set_error("null argument"); return MDFT_E_ARG; }
    *count = h->launches;
    return MDFT_OK;
}

int mdft_get_stage_times(const mdft_handle *h, double *ms5, int *count) {
    if (!h || !ms5) { set_error("null argument"); return MDFT_E_ARG; }
    for (int i = 0; i < ST_COUNT; ++i) ms5[i] = h->stage_ms[i];
    if (count) *count = h->stage_count;
    return MDFT_OK;
}

}  // extern "C"

#include "solve.cuh"
#include "mixture.cuh"
