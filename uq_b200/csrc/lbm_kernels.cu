// CUDA kernels of the D2Q13 thermal LBM step for sm_100a.
//
// One time step of a batch is a short sequence of launches over a packed
// tile list of all samples (see lbm_engine.cu):
//   P0  pointwise stages      (RK3 stages 1+2 -> f2; RK1 stage 1 -> f1;
//                              EULER copies f) into stage buffer 2
//   W   wall fluxes           alpha for every solid node next to fluid
//   P1  stencil + stage       fluxes of buffer 2, divergence, then RK3 stage 3
//                              (-> buffer 3, and the update partial sum in
//                              place of f) or the RK1/EULER update of f
//   W   wall fluxes of buffer 3                        (RK3 only)
//   P2  stencil + update      fluxes of buffer 3, final RK3 combination
// The reference computes the same quantities in RK1/RK3/EULER/EULER_EQ
// (cpuLBM.cpp:1597-2283) with full-field temporaries.
#include "lbm_node.cuh"
#include "tma.cuh"

#include <cuda_runtime.h>

#include <algorithm>

namespace uqlbm {

// ------------------------------------------------------------------- init
// initialiseFunctions (cpuLBM.cpp:846-875) for one node: f, h = equilibrium
// of (rho, ux, uy, T), stored as deviations from the rest state; solid and
// permanent nodes also seed stage buffers 2/3, whose contents never change
// for them.  Returns false when the equilibrium mass check fails.  One
// compiled body serves every initialising kernel, so a state set from
// fields is bit-for-bit the state built at creation.
template <class S>
__device__ __noinline__ bool init_node(double rho, double ux, double uy, double T, const SampleParams &sp,
                                       const double *fr, S *state, S *buf2, S *buf3, long long o, bool fixed)
{
    EqState<double> q = eq_state<double>(rho, ux, uy, T / sp.Tc, sp);
    double f[NQ], h[NQ];
    eq_all(q, f, h);
    double sf = 0;
    for (int i = 0; i < NQ; ++i) sf += f[i];
    for (int i = 0; i < NQ; ++i) {
        const long long k = (long long)i * sp.plane + o;
        const Pair<S> v = make_pair2((S)(f[i] - fr[i]), (S)(h[i] - fr[NQ + i]));
        pair_base(state, sp)[k] = v;
        if (fixed) {
            pair_base(buf2, sp)[k] = v;
            pair_base(buf3, sp)[k] = v;
        }
    }
    return !(fabs(sf - rho) > 1e-6);
}

// ------------------------------------------------------------------- P0
// RK: 1 (RK3 stages 1+2), 0 (RK1 stage 1), 2 (EULER / EULER_EQ: copy).
// Pointwise.  A node's 13 pairs are loaded once and stay in registers for the
// moments and for the stages; the stage values of nodes near an x edge of a
// sample with ghost columns are stored at their periodic images too.  Bound
// by memory latency at 24 (FP64 16) warps per SM: 3.5 M nodes in 169 us, 67 %
// of the copy rate (FP64 271 us, 83 %); 64 registers and four blocks, or
// loading the state twice, are 4 % and 17 % slower.
template <class S>
struct Stage0Blocks {
    static constexpr int value = sizeof(S) == 4 ? 3 : 2;
};
template <class S, int RK, bool LAW>
__global__ void __launch_bounds__(256, Stage0Blocks<S>::value) k_stage0(KArgs<S> a)
{
    using C = S;
    using V = Pair<S>;
    const Tile t = a.tiles[blockIdx.x];
    const SampleParams &sp = a.samples[t.sample];
    const int x = t.x0 + threadIdx.x % a.tx, y = t.y0 + threadIdx.x / a.tx;
    if (x >= sp.nx || y >= sp.ny) return;
    const int o = y * sp.pitch + x, PL = (int)sp.plane;
    const long long node = sp.node_off + o;
    const int type = a.nflags[node] & NF_TYPE;
    pdl_wait();
    if (type != 0) return;
    const V *__restrict__ st = pair_base(a.state, sp) + o;
    V *__restrict__ b2 = pair_base(a.buf2, sp) + o;
    const int gd = a.phased ? 0 : ghost_offset(sp, x);
    V v[NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i) v[i] = st[i * PL];
    if constexpr (RK >= 2) {  // EULER, EULER_EQ: fluxes of the state itself
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            b2[i * PL] = v[i];
            if (gd) b2[i * PL + gd] = v[i];
        }
        if (a.want_residual) a.told[node] = node_macro_rd<false>([&](int i) { return v[i]; }, sp).T;
        return;
    }
    const Macro m = node_macro_rd<LAW>([&](int i) { return v[i]; }, sp);
    pdl_trigger();
    if (a.want_residual) a.told[node] = m.T;
    const bool bad = first_stage<S, RK == 1 ? 1 : 0>(v, m, sp, a.eq_tol, [&](int i, V nv) {
        b2[i * PL] = nv;
        if (gd) b2[i * PL + gd] = nv;
    });
    if (bad) atomicOr(&a.status[t.sample], STATUS_EQ);
}

// -------------------------------------------------------------------- W
template <class S, class C>
__global__ void k_wall(KArgs<S> a, const S *__restrict__ stage, const WallNode *__restrict__ walls, int nwalls)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nwalls) return;
    const WallNode w = walls[k];
    const SampleParams sp = a.samples[w.sample];
    const StageView<S> v{stage + sp.state_off, a.nflags + sp.node_off, (int)sp.plane, sp.pitch};
    const double am1 = wall_alpha_m1<S, C>(sp, v, w.x, w.y, a.dxv[sp.xoff + w.x], a.dyv[sp.yoff + w.y],
                                           a.fref + NPL * w.sample);
    a.template alpha_as<C>()[sp.node_off + (long long)w.y * sp.pitch + w.x] = (C)am1;
}

// Ghost columns (SampleParams::gx): block (s, i) copies, in every row of
// plane i of sample s0 + s, the gx columns at each x edge of the domain to
// the ghost columns beyond the other edge: x in [-gx, 0) gets x + nx, x in
// [nx, nx + gx) gets x - nx.  The stepping kernels keep the ghosts of the
// values they write; this refreshes them after the state is set from
// outside (the fixed nodes' stage values change there).
template <class S>
__global__ void k_fill_ghosts(const SampleParams *samples, int s0, S *buf)
{
    const SampleParams &sp = samples[s0 + blockIdx.x];
    if (!sp.gx) return;  // else GHOST_X
    constexpr int gx = GHOST_X, w = 2 * GHOST_X;
    const int nx = sp.nx, n = sp.ny * w, pitch = sp.pitch;
    Pair<S> *pl = pair_base(buf, sp) + (long long)blockIdx.y * sp.plane;
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const int y = e / w, c = e % w;
        const int xg = c < gx ? c - gx : nx + (c - gx);  // the ghost
        Pair<S> *row = pl + (long long)y * pitch;
        row[xg] = row[c < gx ? xg + nx : c - gx];        // its image in the domain
    }
}

template <class S>
cudaError_t launch_fill_ghosts(const SampleParams *samples, int s0, int ns, S *buf2, S *buf3, cudaStream_t st)
{
    if (ns > 0) {
        if (buf2) k_fill_ghosts<S><<<dim3(ns, NQ), 256, 0, st>>>(samples, s0, buf2);
        if (buf3) k_fill_ghosts<S><<<dim3(ns, NQ), 256, 0, st>>>(samples, s0, buf3);
    }
    return cudaGetLastError();
}
template cudaError_t launch_fill_ghosts<double>(const SampleParams *, int, int, double *, double *, cudaStream_t);
template cudaError_t launch_fill_ghosts<float>(const SampleParams *, int, int, float *, float *, cudaStream_t);

// per-sample residual = sqrt(sum / (Nx Ny)) (runOne, cpuLBM.cpp:2322-2331):
// block s adds sample s's per-tile sums, thread t every 256th, then the
// threads pairwise (always the same order).  One thread per sample took
// 0.62 ms over the 16,384 tiles of a 2048 x 2048 grid, more than the step.
__global__ void __launch_bounds__(256) k_residual(const SampleParams *samples, const double *partial, const int *tile_first,
                                                  const int *tile_count, double *residual)
{
    __shared__ double sum[256];
    const int s = blockIdx.x, t = threadIdx.x, n = tile_count[s];
    const double *p = partial + tile_first[s];
    double v = 0;
    for (int k = t; k < n; k += 256) v += p[k];
    sum[t] = v;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (t < w) sum[t] += sum[t + w];
        __syncthreads();
    }
    if (t == 0) residual[s] = sqrt(sum[0] / ((double)samples[s].nx * samples[s].ny));
}

// ------------------------------------------------------------ boundary I/O
// Fields at the boundary are in the reference's [x*Ny + y] order, y fastest;
// the planes have x fastest.  A block moves tiles of 32 columns x 8 rows
// through shared memory, so that both sides are read and written in whole
// sectors (8 values along y are 64 bytes; a thread per boundary value touched
// a sector of every plane for 8 bytes of it).  Blocks (., j) take sample
// s0 + j; with `all`, a sample's fields start SampleParams::lat_off values in.
constexpr int IO_X = 32, IO_Y = 8, IO_N = IO_X * IO_Y;

template <class F>
__device__ __forceinline__ void io_tiles(const SampleParams &sp, F f)
{
    const int ntx = (sp.nx + IO_X - 1) / IO_X, nt = ntx * ((sp.ny + IO_Y - 1) / IO_Y);
    for (int q = blockIdx.x; q < nt; q += gridDim.x) f(q % ntx * IO_X, q / ntx * IO_Y);
}

// macroPropShort of every node: rho, ux, uy, T, p, each `stride` values apart
template <class S>
__global__ void __launch_bounds__(IO_N) k_macro_out(const SampleParams *samples, int s0, int all, const S *state, double *out,
                                                    long long stride)
{
    __shared__ double buf[5][IO_Y][IO_X + 1];
    const SampleParams &sp = samples[s0 + blockIdx.y];
    const int t = threadIdx.x;
    if (all) out += sp.lat_off;
    io_tiles(sp, [&](int x0, int y0) {
        {
            const int lx = t % IO_X, ly = t / IO_X, x = x0 + lx, y = y0 + ly;
            if (x < sp.nx && y < sp.ny) {
                const Macro m = node_macro<S>(pair_base(state, sp), sp, (long long)y * sp.pitch + x);
                const double v[5] = {m.rho, m.ux, m.uy, m.T, m.p};
#pragma unroll
                for (int k = 0; k < 5; ++k) buf[k][ly][lx] = v[k];
            }
        }
        __syncthreads();
        const int lx = t / IO_Y, ly = t % IO_Y, x = x0 + lx, y = y0 + ly;
        if (x < sp.nx && y < sp.ny) {
#pragma unroll
            for (int k = 0; k < 5; ++k) out[k * stride + (long long)x * sp.ny + y] = buf[k][ly][lx];
        }
        __syncthreads();
    });
}

// planes <-> reference AoS [(x*Ny + y)*13 + i] in FP64, f then h, of sample s
template <class S>
__global__ void __launch_bounds__(IO_N) k_dist_io(const SampleParams *samples, int s, S *state, S *buf2, S *buf3, double *aos,
                                                  int to_aos, const uint8_t *nflags, const double *fref)
{
    __shared__ double buf[IO_X][IO_Y * NQ + 1];
    const double *fr = fref + NPL * s;
    const SampleParams &sp = samples[s];
    const long long n = (long long)sp.nx * sp.ny * NQ;
    const int t = threadIdx.x, lx = t % IO_X, ly = t / IO_X;
    io_tiles(sp, [&](int x0, int y0) {
        const int x = x0 + lx, y = y0 + ly;
        const bool in = x < sp.nx && y < sp.ny;
        const long long o = (long long)y * sp.pitch + x;
        const int rows = min(IO_Y, sp.ny - y0) * NQ;  // values of a column of the tile
        Pair<S> v[NQ];
        if (to_aos && in) {
#pragma unroll
            for (int i = 0; i < NQ; ++i) v[i] = pair_base(state, sp)[(long long)i * sp.plane + o];
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            double *a = aos + half * n;
            auto move = [&](auto one) {
                for (int k = t; k < IO_X * IO_Y * NQ; k += IO_N) {
                    const int c = k / (IO_Y * NQ), r = k % (IO_Y * NQ);
                    if (x0 + c < sp.nx && r < rows) one(a[((long long)(x0 + c) * sp.ny + y0) * NQ + r], buf[c][r]);
                }
            };
            if (to_aos) {
                if (in) {
#pragma unroll
                    for (int i = 0; i < NQ; ++i) buf[lx][ly * NQ + i] = (double)(half ? v[i].y : v[i].x) + fr[half * NQ + i];
                }
                __syncthreads();
                move([](double &g, double &b) { g = b; });
            } else {
                move([](double &g, double &b) { b = g; });
                __syncthreads();
                if (in) {
#pragma unroll
                    for (int i = 0; i < NQ; ++i) {
                        const S w = (S)(buf[lx][ly * NQ + i] - fr[half * NQ + i]);
                        if (half) v[i].y = w;
                        else v[i].x = w;
                    }
                }
            }
            __syncthreads();
        }
        if (!to_aos && in) {
            const bool fixed = (nflags[sp.node_off + o] & NF_TYPE) != 0;  // fixed nodes seed the stage buffers
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                const long long e = (long long)i * sp.plane + o;
                pair_base(state, sp)[e] = v[i];
                if (fixed) {
                    pair_base(buf2, sp)[e] = v[i];
                    pair_base(buf3, sp)[e] = v[i];
                }
            }
        }
    });
}

// f, h = equilibria of per-node fields (FP64): rho, ux, uy, T, each `stride`
// values apart
template <class S>
__global__ void __launch_bounds__(IO_N) k_set_macro(const SampleParams *samples, int s0, int all, S *state, S *buf2, S *buf3,
                                                    const double *fields, long long stride, const uint8_t *nflags,
                                                    const double *fref)
{
    __shared__ double buf[4][IO_Y][IO_X + 1];
    const int s = s0 + blockIdx.y, t = threadIdx.x;
    const double *fr = fref + NPL * s;
    const SampleParams &sp = samples[s];
    if (all) fields += sp.lat_off;
    if (!stride) {  // the samples' four fields together
        fields += 4 * sp.lat_off - (all ? sp.lat_off : 0);
        stride = (long long)sp.nx * sp.ny;
    }
    io_tiles(sp, [&](int x0, int y0) {
        {
            const int lx = t / IO_Y, ly = t % IO_Y, x = x0 + lx, y = y0 + ly;
            if (x < sp.nx && y < sp.ny) {
#pragma unroll
                for (int k = 0; k < 4; ++k) buf[k][ly][lx] = fields[k * stride + (long long)x * sp.ny + y];
            }
        }
        __syncthreads();
        const int lx = t % IO_X, ly = t / IO_X, x = x0 + lx, y = y0 + ly;
        if (x < sp.nx && y < sp.ny) {
            const long long o = (long long)y * sp.pitch + x;
            const bool fixed = (nflags[sp.node_off + o] & NF_TYPE) != 0;
            init_node<S>(buf[0][ly][lx], buf[1][ly][lx], buf[2][ly][lx], buf[3][ly][lx], sp, fr, state, buf2, buf3, o, fixed);
        }
        __syncthreads();
    });
}

// calls f(grid, first sample) for ns samples of up to `nodes` nodes each, as
// many in one launch as a grid holds along y
template <class F>
static cudaError_t io_launches(long long nodes, int s0, int ns, F f)
{
    const long long tiles = (nodes + IO_N - 1) / IO_N + 1;
    const unsigned x = (unsigned)std::min<long long>(tiles, ns > 1 ? 256 : 2048);
    constexpr int MAX_Y = 65535;
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < ns && e == cudaSuccess; k += MAX_Y) {
        f(dim3(x, (unsigned)std::min(MAX_Y, ns - k)), s0 + k);
        e = cudaGetLastError();
    }
    return e;
}

template <class S>
cudaError_t launch_set_macro(const SampleParams *samples, int s0, int ns, S *state, S *buf2, S *buf3, const double *fields,
                             long long stride, const uint8_t *nflags, const double *fref, long long nodes, cudaStream_t st)
{
    return io_launches(nodes, s0, ns, [&](dim3 grid, int s) {
        k_set_macro<S><<<grid, IO_N, 0, st>>>(samples, s, ns > 1, state, buf2, buf3, fields, stride, nflags, fref);
    });
}
template cudaError_t launch_set_macro<double>(const SampleParams *, int, int, double *, double *, double *, const double *,
                                              long long, const uint8_t *, const double *, long long, cudaStream_t);
template cudaError_t launch_set_macro<float>(const SampleParams *, int, int, float *, float *, float *, const double *,
                                             long long, const uint8_t *, const double *, long long, cudaStream_t);

// ----------------------------------------------------------------- launchers
// phase: 0 pointwise stages, 1 stencil phase over buffer 2, 2 RK3 final
// stencil phase over buffer 3, 3/4 wall fluxes of buffer 2/3.  rk selects
// the method of the tiles passed (one method per launch).
template <class S, class C>
cudaError_t launch_phase(const KArgs<S> &a, int phase, int rk, const Tile *tiles, int ntiles, const WallNode *walls,
                         int nwalls, cudaStream_t st, int path)
{
    KArgs<S> k = a;
    k.tiles = tiles;
    k.ntiles = ntiles;
    const int NT = a.tx * a.ty;
    if (phase == 0) {
        if (!ntiles) return cudaSuccess;
        return launch_step_kernel(rk >= 2         ? k_stage0<S, 2, false>
                                  : k.constant_mu ? (rk ? k_stage0<S, 1, sizeof(S) == 4> : k_stage0<S, 0, sizeof(S) == 4>)
                                                  : (rk ? k_stage0<S, 1, true> : k_stage0<S, 0, true>),
                                  ntiles, NT, 0, st,
                                  !k.phased, k);
    } else if (phase == 1 || phase == 2) {
        if (!ntiles) return cudaSuccess;
        const int mode = phase == 2 ? 2 : (rk == 1 ? 1 : (rk == 0 ? 3 : (rk == 2 ? 4 : 5)));
        return launch_flux<S>(mode, k, ntiles, path, st);
    } else if (phase == 3 || phase == 4) {
        if (nwalls) k_wall<S, C><<<(nwalls + 127) / 128, 128, 0, st>>>(k, phase == 3 ? a.buf2 : a.buf3, walls, nwalls);
    }
    return cudaGetLastError();
}

template <class S, class C>
cudaError_t prepare_kernels()
{
    return prepare_flux<S>();
}

template <class S>
cudaError_t launch_macro_out(const SampleParams *samples, int s0, int ns, const S *state, double *out, long long stride,
                             long long nodes, cudaStream_t st)
{
    return io_launches(nodes, s0, ns, [&](dim3 grid, int s) {
        k_macro_out<S><<<grid, IO_N, 0, st>>>(samples, s, ns > 1, state, out, stride);
    });
}

template <class S>
cudaError_t launch_dist_io(const SampleParams *samples, int s, S *state, S *buf2, S *buf3, double *aos, int to_aos,
                           const uint8_t *nflags, const double *fref, long long nodes, cudaStream_t st)
{
    return io_launches(nodes, s, 1, [&](dim3 grid, int k) {
        k_dist_io<S><<<grid, IO_N, 0, st>>>(samples, k, state, buf2, buf3, aos, to_aos, nflags, fref);
    });
}

// Self-test of the bounded mbarrier wait the stencil kernels use: one block
// initialises a barrier that expects one arrival and waits on it with the
// same poll limit.  With arrive = 0 nothing arrives, the wait runs out and
// the block records STATUS_TIMEOUT and returns; with arrive = 1 thread 0
// arrives first and the wait succeeds.  No copy is ever in flight.
__global__ void k_wait_selftest(int *status, int arrive, uint32_t polls)
{
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0 && arrive) mbar_arrive_expect_tx(&bar, 0);
    __syncthreads();
    const bool ok = mbar_wait_bounded(&bar, 0, polls);
    if (!ok && threadIdx.x == 0) atomicOr(status, STATUS_TIMEOUT);
}

cudaError_t launch_wait_selftest(int *status, int arrive, cudaStream_t st)
{
    k_wait_selftest<<<1, 32, 0, st>>>(status, arrive, TMA_WAIT_POLLS);
    return cudaGetLastError();
}

cudaError_t launch_residual(const SampleParams *samples, int nsamples, const double *partial, const int *tile_first,
                            const int *tile_count, double *residual, cudaStream_t st)
{
    k_residual<<<nsamples, 256, 0, st>>>(samples, partial, tile_first, tile_count, residual);
    return cudaGetLastError();
}

template cudaError_t launch_phase<double, double>(const KArgs<double> &, int, int, const Tile *, int, const WallNode *,
                                                  int, cudaStream_t, int);
template cudaError_t launch_phase<float, float>(const KArgs<float> &, int, int, const Tile *, int, const WallNode *, int,
                                                cudaStream_t, int);
template cudaError_t prepare_kernels<double, double>();
template cudaError_t prepare_kernels<float, float>();
template cudaError_t launch_macro_out<double>(const SampleParams *, int, int, const double *, double *, long long, long long,
                                              cudaStream_t);
template cudaError_t launch_macro_out<float>(const SampleParams *, int, int, const float *, double *, long long, long long,
                                             cudaStream_t);
template cudaError_t launch_dist_io<double>(const SampleParams *, int, double *, double *, double *, double *, int,
                                            const uint8_t *, const double *, long long, cudaStream_t);
template cudaError_t launch_dist_io<float>(const SampleParams *, int, float *, float *, float *, double *, int,
                                           const uint8_t *, const double *, long long, cudaStream_t);

}  // namespace uqlbm
