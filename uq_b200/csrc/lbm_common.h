// Host-side pieces shared by batches (lbm_engine.cu) and the request server
// (lbm_server.cu): device buffers, the derived per-sample description, the
// per-sample preparation that does not depend on where a sample is packed,
// and the launch sequence of one step over packed tile and wall lists.
#pragma once

#include "lbm_device.cuh"
#include "lbm_host.h"
#include "lbm_kernels.h"
#include "../../include/uq_lbm.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <memory>
#include <vector>

namespace uqlbm {

template <class T>
struct DevBuf {
    T *p = nullptr;
    size_t n = 0;    // elements in use
    size_t cap = 0;  // elements allocated
    void alloc(size_t count)
    {
        free();
        if (count == 0) return;
        CU(cudaMalloc(&p, count * sizeof(T)));
        n = cap = count;
    }
    void upload(const std::vector<T> &v, cudaStream_t s)
    {
        alloc(v.size());
        if (!v.empty()) CU(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    }
    // keep the allocation when it is large enough (grows by half again
    // otherwise), so repeated repacks do not reallocate
    void upload_keep(const std::vector<T> &v, cudaStream_t s)
    {
        if (v.size() > cap) {
            const size_t c = std::max(v.size(), cap + cap / 2);
            free();
            CU(cudaMalloc(&p, c * sizeof(T)));
            cap = c;
        }
        n = v.size();
        if (!v.empty()) CU(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    }
    void free()
    {
        if (p) cudaFree(p);
        p = nullptr;
        n = cap = 0;
    }
    ~DevBuf() { free(); }
};

// Host-side description of one sample after refineInput / setupVars.
struct HostSample {
    int nx = 0, ny = 0, rk = 1, fm = 1;
    int flags = 0;
    double R = 1, b = 5, K = 3, Tc = 1, c = 1, mu = 0, Pr = 1, dt = 0, tol = 0;
    double rho_ref = 1, T_ref = 1;  // completed reference state (refineInput)
    double gamma = 1.4;
    int mu_model = 0;               // viscosity law (lbm_config::mu_model)
    double upsilon = 0, S_v = 0;
    int nsteps = 0;
    std::vector<double> dx, dy;
    std::vector<uint8_t> type;  // [y*nx + x]
    // initial node state rho, ux, uy, T, each nx ny values in the boundary's
    // [x*ny + y] order (freed once on the device)
    std::unique_ptr<double[]> fields;
    // driver state (cpuLBM::step, residual, initRes, resNorm; main.cpp:34-70)
    int step = 0;
    double residual = 1, resNorm = 0, initRes[100] = {0};
};

// whether no sample has a viscosity law (KArgs::constant_mu)
inline bool constant_mu(const std::vector<SampleParams> &sp)
{
    return std::all_of(sp.begin(), sp.end(), [](const SampleParams &p) { return p.visc == 0; });
}

// What a sample needs on the device apart from its place in a packing.
struct PreparedSample {
    SampleParams p{};  // offsets, first_tile and ntile are set when packed
    double fref[NPL] = {};
    std::vector<uint8_t> flags;  // node flags, ny rows of pitch bytes
    std::vector<WallNode> walls; // solid nodes next to fluid; sample field 0
    std::vector<double> tdx, tdy, dx, dy;
};

HostSample derive(const lbm_config &c, const lbm_init &in);
void prepare_sample(const HostSample &h, int prec, PreparedSample &out);
// append the tx x ty tiles of one sample (p: its parameters; flags in pitch
// layout) with the given sample index, each with its kind (see Tile); gid
// numbers continue from out.size()
void cut_tiles(const uint8_t *flags, const SampleParams &p, int tx, int ty, int sample, std::vector<Tile> &out);
// the wall nodes whose factor a general tile of the sample reads (sweep tiles
// form the factors of straight walls themselves); tiles: the sample's, as
// cut_tiles made them
void needed_walls(const SampleParams &p, int tx, int ty, const Tile *tiles, const std::vector<WallNode> &walls,
                  std::vector<WallNode> &out);
// TMA descriptors of one sample (MAPS_PER_SAMPLE of them)
void encode_stage_maps(int prec, const SampleParams &p, unsigned char *buf2, unsigned char *buf3, int tx, int ty,
                       CUtensorMap *maps);
void check_tile_shape(int x, int y);
int round_up(int v, int m);

// A run of tiles in a device list.
struct TileRun {
    const Tile *p = nullptr;
    int n = 0;
};

// Device pointers and lengths of the packed lists one step launches over.
// The pointwise phase runs over the tiles of each RKMETHOD in sample order;
// the stencil phases over the same tiles as two runs, the sweep tiles and
// the general tiles, one kernel per run.
struct StepLists {
    TileRun pointwise[4];            // tiles by RKMETHOD, sample order
    TileRun sweep[4], general[4];    // the same tiles by kind
    TileRun rk3_sweep, rk3_general;  // RK3 tiles (final stencil phase)
    // the wall nodes that general tiles read (WallNode lists)
    const WallNode *walls_all = nullptr, *walls_rk3 = nullptr;
    int n_walls_all = 0, n_walls_rk3 = 0;
    // for a step taken phase by phase: the sweep runs' kinds (tile_rank: 0,
    // 1, the rest 2), every wall node, and the samples
    int kinds[4][2] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}}, rk3_kinds[2] = {0, 0};
    const WallNode *every_wall = nullptr, *every_wall_rk3 = nullptr;
    int n_every_wall = 0, n_every_wall_rk3 = 0;
    const SampleParams *samples = nullptr;
    int nsamples = 0;
    bool any_ghost = false;
};

// A device list of n tiles whose first ns are sweep tiles, as two runs.
inline void split_runs(const Tile *p, int n, int ns, TileRun &sweep, TileRun &general)
{
    sweep.p = p;
    sweep.n = ns;
    general.p = p ? p + ns : nullptr;
    general.n = n - ns;
}

// Reorder a host tile list by kind (tile_rank; each kind keeps its order);
// ns: how many are sweep tiles, kinds: how many of the first two kinds.
inline void order_by_kind(std::vector<Tile> &v, int &ns, int *kinds = nullptr)
{
    std::stable_sort(v.begin(), v.end(), [](const Tile &a, const Tile &b) { return tile_rank(a) < tile_rank(b); });
    int n[4] = {0, 0, 0, 0};
    for (const Tile &t : v) ++n[tile_rank(t)];
    ns = n[0] + n[1] + n[2];
    if (kinds) {
        kinds[0] = n[0];
        kinds[1] = n[1];
    }
}

template <class S, class C>
void stencil_runs(const KArgs<S> &a, int phase, int m, const TileRun &s, const TileRun &g, cudaStream_t st)
{
    if (s.n) CU((launch_phase<S, C>(a, phase, m, s.p, s.n, nullptr, 0, st, FLUX_SWEEP)));
    if (g.n) CU((launch_phase<S, C>(a, phase, m, g.p, g.n, nullptr, 0, st, FLUX_GENERAL)));
}

// n steps: pointwise stages, first stencil phase, and for RK3 the final
// stencil phase; wall factors before a stencil phase with general tiles that
// read some.  Where steps are joined, RK3's final phase forms the next step's
// pointwise stages, so that only the first step launches them.
template <class S, class C>
void enqueue_steps(KArgs<S> a, const StepLists &l, int n, cudaStream_t st)
{
    const bool join = joins<S>(a.tx, a.ty);
    const bool rk3 = l.rk3_sweep.n || l.rk3_general.n;
    for (int k = 0; k < n; ++k) {
        for (int m = 0; m < 4; ++m)
            if (l.pointwise[m].n && !(join && m == 1 && k)) CU((launch_phase<S, C>(a, 0, m, l.pointwise[m].p, l.pointwise[m].n, nullptr, 0, st)));
        CU((launch_phase<S, C>(a, 3, 0, nullptr, 0, l.walls_all, l.n_walls_all, st)));
        for (int m = 0; m < 4; ++m) stencil_runs<S, C>(a, 1, m, l.sweep[m], l.general[m], st);
        if (!rk3) continue;
        CU((launch_phase<S, C>(a, 4, 1, nullptr, 0, l.walls_rk3, l.n_walls_rk3, st)));
        a.next = join && k + 1 < n;
        stencil_runs<S, C>(a, 2, 1, l.rk3_sweep, l.rk3_general, st);
    }
}

// kernels that enqueue_steps launches
inline int steps_launches(const StepLists &l, int n, bool join)
{
    int per = l.n_walls_all ? 1 : 0;
    for (int m = 0; m < 4; ++m) per += (l.pointwise[m].n ? 1 : 0) + (l.sweep[m].n ? 1 : 0) + (l.general[m].n ? 1 : 0);
    if (l.rk3_sweep.n || l.rk3_general.n)
        per += (l.n_walls_rk3 ? 1 : 0) + (l.rk3_sweep.n ? 1 : 0) + (l.rk3_general.n ? 1 : 0);
    return n * per - (join && n > 0 && l.pointwise[1].n ? n - 1 : 0);
}

// The same step phase by phase, every part in launches of its own (the ghost
// columns, the wall factors, each kind of tile): what lbm_batch_profile times
// and a batch without a graph runs.  Same results, bit for bit.  ev
// (optional) receives events [0] start, after pointwise, walls 2, phase 1,
// walls 3, phase 2.
template <class S, class C>
void enqueue_step_phased(KArgs<S> a, const StepLists &l, cudaStream_t st, cudaEvent_t *ev = nullptr)
{
    a.phased = 1;
    auto kinds = [&](int phase, int m, const TileRun &s, const int *k, const TileRun &g) {
        const TileRun run[3] = {{s.p, k[0]}, {s.p + k[0], k[1]}, {s.p + k[0] + k[1], s.n - k[0] - k[1]}};
        for (const TileRun &r : run) stencil_runs<S, C>(a, phase, m, r, TileRun{}, st);
        stencil_runs<S, C>(a, phase, m, TileRun{}, g, st);
    };
    if (ev) CU(cudaEventRecord(ev[0], st));
    for (int m = 0; m < 4; ++m)
        if (l.pointwise[m].n) CU((launch_phase<S, C>(a, 0, m, l.pointwise[m].p, l.pointwise[m].n, nullptr, 0, st)));
    if (l.any_ghost) CU(launch_fill_ghosts<S>(l.samples, 0, l.nsamples, a.buf2, nullptr, st));
    if (ev) CU(cudaEventRecord(ev[1], st));
    CU((launch_phase<S, C>(a, 3, 0, nullptr, 0, l.every_wall, l.n_every_wall, st)));
    if (ev) CU(cudaEventRecord(ev[2], st));
    for (int m = 0; m < 4; ++m) kinds(1, m, l.sweep[m], l.kinds[m], l.general[m]);
    if (ev) CU(cudaEventRecord(ev[3], st));
    const bool rk3 = l.rk3_sweep.n || l.rk3_general.n;
    if (rk3) CU((launch_phase<S, C>(a, 4, 1, nullptr, 0, l.every_wall_rk3, l.n_every_wall_rk3, st)));
    if (ev) CU(cudaEventRecord(ev[4], st));
    if (rk3) kinds(2, 1, l.rk3_sweep, l.rk3_kinds, l.rk3_general);
    if (ev) CU(cudaEventRecord(ev[5], st));
}

// kernels that enqueue_step_phased launches
inline int phased_launches(const StepLists &l)
{
    auto kinds = [](const TileRun &s, const int *k, const TileRun &g) {
        return (k[0] ? 1 : 0) + (k[1] ? 1 : 0) + (s.n > k[0] + k[1] ? 1 : 0) + (g.n ? 1 : 0);
    };
    int n = (l.any_ghost ? 1 : 0) + (l.n_every_wall ? 1 : 0);
    for (int m = 0; m < 4; ++m) n += (l.pointwise[m].n ? 1 : 0) + kinds(l.sweep[m], l.kinds[m], l.general[m]);
    if (l.rk3_sweep.n || l.rk3_general.n)
        n += (l.n_every_wall_rk3 ? 1 : 0) + kinds(l.rk3_sweep, l.rk3_kinds, l.rk3_general);
    return n;
}

}  // namespace uqlbm
