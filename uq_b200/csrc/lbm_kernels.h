// Host-visible kernel interface of the D2Q13 LBM step (see lbm_kernels.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace uqlbm {

struct SampleParams;
struct Tile;

constexpr int STATUS_EQ = 1;         // equilibrium mass check (cpuLBM.cpp:839-843)
constexpr int STATUS_NONFINITE = 2;  // NaN / Inf / rho <= 0 in the state
constexpr int STATUS_TIMEOUT = 4;    // a bounded device-side wait ran out

// tensor maps per sample: the stage buffers 2 and 3, each with the stencil
// kernels' three box shapes (x lines, y lines, both; see lbm_box.h)
constexpr int MAPS_PER_SAMPLE = 6;
// the default tile shape, also compiled into the stencil kernels (box
// widths, strides and the thread-to-line map become constants); other shapes
// run kernels with the shape read at run time.  Of a 32 x 8 tile, the lines
// of one direction along either axis are one warp's work (see lbm_flux.cuh).
constexpr int TILE_CX = 32, TILE_CY = 8;

// Whether RK3 steps in a row are joined (the final phase of one forms stages 1
// and 2 of the next: the state is not read again, 104 of 936 bytes a node).
// FP32 gains 3 % on large batches and nothing on the smallest.  FP64 would
// gain 2 % and lose 6 % at 64 x 128, where the longer kernel is a longer
// chain; RK1 has one stencil phase, which would have to fill a buffer that it
// does not read, and loses 5 % to spills.
template <class S>
constexpr bool joins(int tx, int ty)
{
    return sizeof(S) == 4 && tx == TILE_CX && ty == TILE_CY;
}

struct WallNode {
    int sample, x, y, pad;
};

// Everything a phase kernel needs, passed by value.
template <class S>
struct KArgs {
    const SampleParams *samples;
    const Tile *tiles;
    int ntiles;
    int tx, ty;  // tile shape (threads = tx * ty)
    S *state;    // f, h (and, between P1 and P2 of RK3, the update partial sum)
    S *buf2;     // stage buffer 2 (f1 or f2)
    S *buf3;     // stage buffer 3 (f3)
    const uint8_t *nflags;
    void *alpha_raw;  // per node: wall correction factor alpha - 1
    double *told;     // T at the start of the step (residual)
    double *partial;  // per-tile residual partial sums
    int *status;      // per-sample status bits
    const double *tdx, *tdy, *dxv, *dyv;
    const CUtensorMap *tmaps;  // per sample MAPS_PER_SAMPLE maps: [buffer 2, buffer 3][box shape]
    int slots;                 // boxes resident at a time (other tile shapes)
    const double *fref;        // per sample: 26 rest-state values subtracted from the stored state
    int want_residual;
    // phases launched apart (enqueue_step_phased): the pointwise kernel leaves
    // the ghost columns to k_fill_ghosts, and straight walls take their
    // factors from k_wall
    int phased;
    // RK3's final phase also forms the next step's stages 1 and 2
    int next;
    int constant_mu;  // no sample has a viscosity law
    double eq_tol;
#ifdef __CUDACC__
    // alpha is stored in the compute type of the kernel instantiation
    template <class C>
    __device__ __forceinline__ C *alpha_as() const { return reinterpret_cast<C *>(alpha_raw); }
#endif
};

// Programmatic dependent launch: a kernel of a step starts while the one
// before it drains, and waits (pdl_wait) before it touches what that one
// writes; until then it reads only what no step changes (tiles, sample
// parameters, node flags).  A launch gap and a block's first look-ups are
// most of a small solve's kernel.
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_step_kernel(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t st, bool overlap,
                               A... args)
{
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}
#endif

// Which tiles a stencil-phase launch covers: the sweep tiles or the general
// tiles of its list, one kernel each (see TILE_SWEEP).
enum FluxPath { FLUX_SWEEP = 1, FLUX_GENERAL = 2 };

template <class S, class C>
cudaError_t launch_phase(const KArgs<S> &a, int phase, int rk, const Tile *tiles, int ntiles, const WallNode *walls,
                         int nwalls, cudaStream_t st, int path = FLUX_GENERAL);
template <class S, class C>
cudaError_t prepare_kernels();
// the stencil kernels (lbm_flux_f32.cu, lbm_flux_f64.cu); mode as k_flux's
template <class S>
cudaError_t launch_flux(int mode, const KArgs<S> &a, int ntiles, int path, cudaStream_t st);
template <class S>
cudaError_t prepare_flux();
// boundary I/O of samples s0 .. s0 + ns - 1, `nodes` the most nodes of one;
// fields `stride` values apart, of one sample, or (ns > 1) of every sample
// SampleParams::lat_off values in (set: stride 0, each sample's four fields
// together, 4 lat_off values in)
template <class S>
cudaError_t launch_macro_out(const SampleParams *samples, int s0, int ns, const S *state, double *out, long long stride,
                             long long nodes, cudaStream_t st);
template <class S>
cudaError_t launch_set_macro(const SampleParams *samples, int s0, int ns, S *state, S *buf2, S *buf3, const double *fields,
                             long long stride, const uint8_t *nflags, const double *fref, long long nodes, cudaStream_t st);
template <class S>
cudaError_t launch_dist_io(const SampleParams *samples, int s, S *state, S *buf2, S *buf3, double *aos, int to_aos,
                           const uint8_t *nflags, const double *fref, long long nodes, cudaStream_t st);
cudaError_t launch_wait_selftest(int *status, int arrive, cudaStream_t st);
// copy the edge columns of stage buffers 2 and 3 into the ghost columns
// (SampleParams::gx) of samples s0 .. s0 + ns - 1 (after their state was set)
template <class S>
cudaError_t launch_fill_ghosts(const SampleParams *samples, int s0, int ns, S *buf2, S *buf3, cudaStream_t st);
cudaError_t launch_residual(const SampleParams *samples, int nsamples, const double *partial, const int *tile_first,
                            const int *tile_count, double *residual, cudaStream_t st);

}  // namespace uqlbm
