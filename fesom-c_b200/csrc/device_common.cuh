// Shared device-side definitions of the B200 FESOM-C time step.
//
// Layout in HBM (device order: the reference order, or with sfc_order the
// order of a Hilbert curve through the mesh, every index translated):
//   * 2D node / element fields: one double per entity.
//   * 2D vectors (U_n_2D, UAB, ...): double2 per element (u, v interleaved,
//     as the Fortran (2,E) arrays).
//   * Level fields: [entity][level] with levels contiguous, exactly the
//     Fortran (nsigma-1, N) / (nsigma, N) arrays, so a column is one
//     contiguous run of L (or NS) doubles.
//   * Connectivity: 0-based int4 / int2; absent neighbour / second element
//     of a boundary edge = -1.
//   * Edge scatters of the reference become gathers over CSR lists that are
//     sorted by the reference edge number, so every node / element receives
//     its contributions in the same order as the serial Fortran loop and the
//     FP64 sums are bit-identical (compiled with --fmad=false).
//   * Jc, Jd, Z, zbar (subroutine jacobian, fv_main.F90:1208-1267) are not
//     stored: they are recomputed with the same expressions from the
//     elevation at the last jacobian call (eta_jac) and sigma.  The element
//     quantities Je and the w_cv-weighted Z / zbar, which every element
//     kernel needs at every level, are stored once per jacobian call.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "fesomc_log.h"
#include "fesomc_trig.h"

// FP32 form: the closure's logarithm is the device logf (the FP64 path uses
// fesomc_log, bit-identical with the oracle's).
static __device__ __forceinline__ float fesomc_log(float x) { return logf(x); }

// Each kernel source is compiled twice: with FESOMC_FP32 = 0 into
// fesomc::f64 (the FP64 path, bit-exact with the reference's algorithm) and
// with FESOMC_FP32 = 1 into fesomc::f32 (the precision form: level fields,
// mesh geometry and the 3D arithmetic in FP32; the 2D sub-cycle state in
// FP64).
#ifndef FESOMC_FP32
#define FESOMC_FP32 0
#endif

namespace fesomc {

constexpr double kG64 = 9.8;
constexpr double kPref = 101325.0;   // P_ref, reference atmospheric pressure (fv_var.F90:17)

// Raises (never lowers) a kernel's dynamic shared-memory limit.  The
// attribute belongs to the kernel, and every model instance of the process
// (ensemble members of different level counts, both precision forms)
// launches the same kernels, so one instance must not shrink another's.
template <typename K>
inline cudaError_t raise_smem_limit(K kernel, size_t bytes) {
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, kernel);
    if (e != cudaSuccess) return e;
    if (bytes <= (size_t)a.maxDynamicSharedSizeBytes) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// ---- compensated sums of the energy diagnostic --------------------------------
// running sum s with its rounding errors in c (Neumaier 1974)
struct CompSum {
    double s, c;
    __device__ __forceinline__ void add(double x) {
        const double t = s + x;
        if (fabs(s) >= fabs(x)) c += (s - t) + x;
        else c += (x - t) + s;
        s = t;
    }
    __device__ __forceinline__ void merge(double os, double oc) {
        add(os);
        c += oc;
    }
};
// The three compensated sums of a block of BLOCK threads, merged in a fixed
// tree (lanes of a warp, then the warps), so that the result does not depend
// on timing; thread k < 3 of the block returns sum k.  Bound by the latency
// of dependent FP64 additions: with three threads adding the block's 256
// values one after the other, and the grid's 592, fesomc_energy_device took
// 74 us on 262 k nodes; the trees are 12 and 15 additions deep: 37 us, of
// which the two kernels 10 + 4.5 us.
template <int BLOCK>
__device__ __forceinline__ double block_sum3(CompSum (&v)[3]) {
    constexpr int W = BLOCK / 32;
    __shared__ double sh[3][2][W];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double os = __shfl_down_sync(0xffffffffu, v[k].s, o), oc = __shfl_down_sync(0xffffffffu, v[k].c, o);
            v[k].merge(os, oc);
        }
        if (lane == 0) {
            sh[k][0][warp] = v[k].s;
            sh[k][1][warp] = v[k].c;
        }
    }
    __syncthreads();
    CompSum t{0.0, 0.0};
    if (threadIdx.x < 3) {
#pragma unroll
        for (int w = 0; w < W; ++w) t.merge(sh[threadIdx.x][0][w], sh[threadIdx.x][1][w]);
    }
    return t.s + t.c;
}
// the sums of nparts triples, one block
template <int BLOCK>
__device__ __forceinline__ double block_total3(const double *part, int nparts) {
    CompSum v[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
    for (int b = threadIdx.x; b < nparts; b += BLOCK)
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k].add(part[(size_t)b * 3 + k]);
    return block_sum3<BLOCK>(v);
}

// ---- max/min exactly as the Fortran MAX/MIN of two values -------------------
template <typename T>
__device__ __forceinline__ T dmax(T a, T b) { return a > b ? a : b; }
template <typename T>
__device__ __forceinline__ T dmin(T a, T b) { return a < b ? a : b; }

__host__ __device__ __forceinline__ double2 make_real2(double x, double y) { return make_double2(x, y); }
__host__ __device__ __forceinline__ float2 make_real2(float x, float y) { return make_float2(x, y); }
__host__ __device__ __forceinline__ double4 make_real4(double x, double y, double z, double w) {
    return make_double4(x, y, z, w);
}
__host__ __device__ __forceinline__ float4 make_real4(float x, float y, float z, float w) {
    return make_float4(x, y, z, w);
}

// Launch-shape knobs (fesomc_gpu_tune_*): threads per block of the kernels
// whose results do not depend on the block shape (one thread per entity or
// per (entity, level), grid-stride, no block-level reduction), and entities
// per block of the column kernels (pressure_col, bpg_elem, update3d, wvel),
// and the form of d3_end (1 one thread per column; FP64 2 to 6 tiles of columns
// in shared memory; FP32 2 one thread per column with its arrays in shared
// memory, 3 to 6 a set-up and a sweep kernel).  A value of 0 selects the
// built-in default.  TK_ZEROFILT, TK_VDIFF and TK_IMPLVISC are accepted and
// read by no launch: the kernel is gone, and the sizes choose the forms.
enum TuneKnob : int {
    TK_VELRHS, TK_VELGRAD3D, TK_ADV3, TK_PULS, TK_EL2NODES, TK_P1EDGE, TK_AB3, TK_VELGRAD2D, TK_SSHEDGE,
    TK_SSHNODE, TK_ADV2D, TK_U2D, TK_ROT, TK_ZEROFILT, TK_AB2, TK_MEGRAD, TK_MNGRAD, TK_MEDGE, TK_MH,
    TK_UPWIND, TK_AV, TK_COLUMNS, TK_D3END, TK_VDIFF, TK_IMPLVISC, kTuneKnobs
};

// sbc_do on the device (fesomc_gpu_set_atm_fields): the time-interpolation
// coefficients of the 8 atmospheric fields per node (device order, 8
// consecutive values per node), the device clock, a scratch for the stress
// per node (2 values per node), and the namelist's nm_net_flux and
// nm_prec_coef
struct AtmDev {
    const double *coef_a, *coef_b, *clock;
    double *tau_node;
    int net_flux;
    double prec_coef;
};

// Quotient of a flat (entity, level) index by the level count, a run-time
// value: with s = ceil(log2 d) and m = floor(2^(31+s) / d) + 1, which fits 32
// bits, m d exceeds 2^(31+s) by at most d <= 2^s, so floor(n m / 2^(31+s)) =
// floor(n / d) for every 0 <= n < 2^31 (Granlund and Montgomery 1994).  One
// multiply and a shift per thread instead of the 64-bit division and
// remainder routines: at 1.05 M nodes, 20 layers, FP64, adv3_edge 0.71 ->
// 0.55 ms, puls_elem 0.37 -> 0.25, el2nodes 0.26 -> 0.21, muscl_edge 1.43 ->
// 1.28, the step 18.0 -> 17.2 ms (232 k nodes, FP32: 2.82 -> 2.76 ms).
struct FastDiv {
    unsigned m, s;   // multiplier, s - 1
    __host__ void set(unsigned d) {
        unsigned b = 1;
        while ((1ull << b) < d) ++b;
        m = (unsigned)((1ull << (31 + b)) / d + 1);
        s = b - 1;
    }
    __device__ __forceinline__ int div(unsigned n) const { return (int)(__umulhi(n, m) >> s); }
};

namespace f64 {
using real = double;
using real2 = double2;
using real4 = double4;
#include "dev_struct.inc"
}  // namespace f64
namespace f32 {
using real = float;
using real2 = float2;
using real4 = float4;
#include "dev_struct.inc"
}  // namespace f32

// full-warp mask of the level shuffles (levels on consecutive lanes)
constexpr unsigned kFull = 0xffffffffu;

// grid-stride helper; every flat index of a model lies below 2^31 (checked
// at init: a larger mesh does not fit the device), and a stride below 2^23
#define GRID_LOOP(i, n) for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < (unsigned)(n); \
                             i += gridDim.x * blockDim.x)

// launch helpers (implemented in model.cu)
int grid_for(long long n, int block);
// entities per block of the column kernels (pressure_col, bpg_elem, update3d,
// wvel) where the knob "columns" does not set them
inline int default_columns(int L) {
    if (L <= 80 || L > 106) return 160 / L > 16 ? 16 : 160 / L < 1 ? 1 : 160 / L;
    // one column leaves lanes of its last warp idle: two or three (at most
    // 320 threads) where they leave fewer; 100 layers, 100 k nodes, FP64: wvel
    // 0.402 -> 0.365 ms, bpg_elem 0.438 -> 0.417, FP32 update3d 0.229 -> 0.200
    int best = 1;
    for (int c = 2; c <= 3; ++c)
        if (c * ((best * L + 31) / 32) > best * ((c * L + 31) / 32)) best = c;
    return best;
}

// up to twice b columns and 320 threads, the least that leave the fewest lanes
// of a block's warps idle (24 layers: 8 instead of 6, 144 of 160 threads; 44: 5 instead of 3)
inline int filled_columns(int L, int b) {
    int best = b;
    for (int c = b + 1; c <= 2 * b && c <= 16 && c * L <= 320; ++c)
        if (c * ((best * L + 31) / 32) > best * ((c * L + 31) / 32)) best = c;
    return best;
}

// Programmatic dependent launch: a kernel started with launch_k may be
// resident while the kernel before it on the stream still runs, so that its
// launch latency hides behind that kernel's tail.  Every kernel started this
// way begins with pdl_enter(), which waits until the kernel before has
// completed and its writes are visible, and only then lets the one after be
// launched: at most one kernel waits at a time, and when a kernel passes its
// wait, every earlier kernel of the stream has completed (each of them
// passed its own first).  That rests on the work before being a kernel: the
// first kernel of a step and every other one behind a memset, a copy or a
// graph on its stream is launched plainly (launch_plain; a captured step
// loses nothing by it, its first kernel has none before it).
// Only grids of at most two blocks per SM are started early.  Steps of small
// meshes are bound by launches (697 nodes: 0.353 -> 0.328 ms per step, 16 k
// nodes: 0.488 -> 0.440 ms); the waiting blocks of a large grid take slots
// and cache from the kernel they wait for (1.05 M nodes: 18.2 -> 19.5 ms with
// every kernel started early; 42 k nodes: 1.65 -> 1.74 ms with up to four
// blocks per SM, 1.63 ms with two).
constexpr unsigned kPdlMaxBlocks = 2 * 148;
inline bool early_grid(unsigned blocks) { return blocks <= kPdlMaxBlocks; }
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}
template <typename... P, typename... A>
inline void launch_as(bool early, void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = early && early_grid(grid.x * grid.y) ? 1 : 0;
    (void)cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
template <typename... P, typename... A>
inline void launch_k(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t s, A... args) {
    launch_as(true, kernel, grid, block, smem, s, args...);
}
template <typename... P, typename... A>
inline void launch_plain(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t s, A... args) {
    launch_as(false, kernel, grid, block, smem, s, args...);
}

// Launches a kernel whose blocks of 'threads' take groups of 'per_block'
// entities and stride over them: as many blocks as are resident at once (a
// few more would make a second, mostly empty wave of all the work).
template <typename... P, typename... A>
inline void launch_resident_as(bool early, void (*kernel)(P...), long long count, int per_block, int threads,
                               size_t smem, cudaStream_t s, A... args) {
    const long long blocks = (count + per_block - 1) / per_block;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem) != cudaSuccess || occ < 1) occ = 1;
    launch_as(early, kernel, (unsigned)(blocks < 148LL * occ ? blocks : 148LL * occ), threads, smem, s, args...);
}
template <typename... P, typename... A>
inline void launch_resident(void (*kernel)(P...), long long count, int per_block, int threads, size_t smem,
                            cudaStream_t s, A... args) {
    launch_resident_as(true, kernel, count, per_block, threads, smem, s, args...);
}

}  // namespace fesomc

#if FESOMC_FP32
#define FESOMC_PREC_BEGIN namespace fesomc { namespace f32 {
#else
#define FESOMC_PREC_BEGIN namespace fesomc { namespace f64 {
#endif
#define FESOMC_PREC_END } }

FESOMC_PREC_BEGIN
#include "dev_helpers.inc"
FESOMC_PREC_END
