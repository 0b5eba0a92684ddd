// The stencil phases of the D2Q13 thermal LBM step (sm_100a): fluxes of a
// stage buffer, their divergence, and the stage or update that follows, one
// tile of nodes per block.
//
// A sweep tile (TILE_SWEEP) works line by line.  TMA brings each moving
// direction's halo box of (f, h) pairs into shared memory; a thread then
// takes one line of a direction, 8 nodes along x or along y, reads it once
// and marches over its 9 faces, so that the differences, the smoothness terms
// and each face flux are formed once and shared by the faces and nodes that
// need them (line_diffs).  On the default tile (32 x 8) a direction's x lines
// are 8 rows x 4 segments and its y lines 32 columns: one warp each way.
// Eight warps take the eight directions with an x and the eight with a y
// component, the four diagonals' two together, so a warp owns its boxes: it
// issues their copies, waits for them alone, and leaves the flux differences
// in the box when it has read it.  The only block barrier comes before the
// per-node stage or update.
// What bounds it: see the measurements at k_flux.
#pragma once

#include "lbm_box.h"
#include "lbm_node.cuh"
#include "tma.cuh"

#include <cuda_runtime.h>

namespace uqlbm {

// pairs of a box, padded to 128 bytes
template <class S>
__host__ __device__ constexpr int box_pairs(int shape, int tx, int ty)
{
    constexpr int a = 128 / (2 * (int)sizeof(S));
    return (box_width<S>(shape, tx) * box_height(shape, ty) + a - 1) / a * a;
}

// Flux differences ("parts"): 16 arrays of ty rows of tx + 1 pairs, one per
// direction and axis (the odd row length keeps an x sweep's stores free of
// bank conflicts).
__host__ __device__ constexpr int part_pairs(int tx, int ty)
{
    return (ty * (tx + 1) + 15) / 16 * 16;
}
__host__ __device__ constexpr int part_index(int i, int axis)
{
    return i <= 4 ? i - 1 : i >= 9 ? i - 5 : 8 + 2 * (i - 5) + axis;
}

// Shared memory.  Default tile: the 12 boxes, whose space takes the parts of
// the direction once read, and the x parts of the diagonals apart (their
// boxes are still being swept along y).  Other tile shapes: `slots` boxes at
// a time and all 16 parts apart.  General tiles: the parts only.
struct FluxSmem {
    int slots;        // boxes resident at a time
    int slot_pairs;   // pairs per slot (not the default tile)
    int part_off;     // the parts (default tile: the diagonals' x parts), in pairs
    int wall_off;     // saved wall faces, in pairs
    int bar_off;      // mbarriers, in pairs
    size_t bytes;     // with 128 bytes of base-alignment slack
};

// default tile: pairs before direction i's box
template <class S>
__host__ __device__ constexpr int box_start(int i)
{
    constexpr int X = box_pairs<S>(BOX_X, TILE_CX, TILE_CY), Y = box_pairs<S>(BOX_Y, TILE_CX, TILE_CY),
                  D = box_pairs<S>(BOX_XY, TILE_CX, TILE_CY);
    // x directions 1, 3, 9, 11, y directions 2, 4, 10, 12, diagonals 5-8
    const int k = i - 1;
    return i <= 4 ? (k / 2) * (X + Y) + (k & 1) * X
         : i <= 8 ? 2 * (X + Y) + (i - 5) * D
                  : 2 * (X + Y) + 4 * D + ((i - 9) / 2) * (X + Y) + (k & 1) * X;
}

template <class S>
__host__ __device__ constexpr FluxSmem flux_smem(int tx, int ty, bool def, bool sweep, int slots)
{
    FluxSmem L{};
    const int pb = 2 * (int)sizeof(S);
    int off = 0;
    L.slots = sweep ? slots : 0;
    if (def && sweep) {
        off += box_start<S>(12) + box_pairs<S>(BOX_Y, tx, ty);
        L.part_off = off;
        off += 4 * part_pairs(tx, ty);
    } else {
        L.slot_pairs = box_pairs<S>(BOX_XY, tx, ty) > box_pairs<S>(BOX_X, tx, ty) ? box_pairs<S>(BOX_XY, tx, ty)
                                                                                  : box_pairs<S>(BOX_X, tx, ty);
        off += L.slots * L.slot_pairs;
        L.part_off = off;
        off += 16 * part_pairs(tx, ty);
    }
    L.wall_off = off;
    if (sweep) off += (4 * tx + 15) / 16 * 16;  // [2 walls][4][tx] values of S
    L.bar_off = off;
    L.bytes = (size_t)off * pb + 12 * sizeof(uint64_t) + 128;
    return L;
}

// boxes resident at a time for other tile shapes: as many as leave room for
// two blocks on an SM, else as many as one block can have
template <class S>
__host__ __device__ constexpr int flux_slots(int tx, int ty)
{
    for (int n = 12; n > 1; --n)
        if (flux_smem<S>(tx, ty, false, true, n).bytes <= 110 * 1024) return n;
    for (int n = 4; n > 1; --n)
        if (flux_smem<S>(tx, ty, false, true, n).bytes <= 220 * 1024) return n;
    return 1;
}

template <class S>
size_t flux_smem_bytes_t(int tx, int ty, bool sweep)
{
    const bool def = tx == TILE_CX && ty == TILE_CY;
    return flux_smem<S>(tx, ty, def, sweep, def ? 12 : flux_slots<S>(tx, ty)).bytes;
}

// how a box lies around the tile: row length, column and row of the tile's
// first node
struct BoxPlace {
    int rs, cx, ry;
};
template <class S>
__device__ __forceinline__ BoxPlace box_place(int shape, int tx)
{
    return BoxPlace{box_width<S>(shape, tx), shape == BOX_Y ? 0 : BoxCols<S>::left, shape == BOX_X ? 0 : HALO};
}

// copy direction i's box of the tile (maps: the stage buffer's three, by box
// shape)
template <class S>
__device__ __forceinline__ void issue_box(Pair<S> *dst, const CUtensorMap *maps, int x0, int y0, int gx, int tx, int ty,
                                          int i, uint64_t *bar)
{
    const int sh = box_shape(i);
    const BoxPlace g = box_place<S>(sh, tx);
    mbar_arrive_expect_tx(bar, (uint32_t)(box_width<S>(sh, tx) * box_height(sh, ty) * sizeof(Pair<S>)));
    const int x = x0 + gx - g.cx, y = y0 - g.ry;
    if constexpr (sizeof(S) == 8) {
        if (box_map_4d<S>(tx)) {  // the map's first dimension is the pair
            tma_load_4d(dst, maps + sh, x, y, i, bar);
            return;
        }
        tma_load_3d(dst, maps + sh, 2 * x, y, i, bar);
    } else {
        tma_load_3d(dst, maps + sh, x, y, i, bar);
    }
}

// TILE_FIX tiles: complete direction i's box beyond the domain before it is
// swept (threads id, id + n, ...).  Along x, for the tile's rows, columns
// outside the domain take the periodic image or the edge column (index,
// cpuLBM.cpp:1033-1113: the stencil's positions clamp); along y, for the
// tile's columns, rows outside likewise, and at a straight wall the wall row
// and the rows beyond it take the extrapolation 2 f(1) - f(2) that stencil()
// puts there.  (The wall row's own nodes are solid: their x lines are not
// used.)
template <class S>
__device__ __noinline__ void fix_box(Pair<S> *box, const SampleParams *gsp, const StageView<S> v, const Tile t, int tx,
                                     int ty, int i, int id, int n)
{
    const SampleParams &sp = *gsp;
    const int sh = box_shape(i);
    const BoxPlace g = box_place<S>(sh, tx);
    const int bx0 = t.x0 - g.cx, by0 = t.y0 - g.ry;  // domain place of the box's first cell
    const bool px = (sp.flags & SF_PERX) != 0, py = (sp.flags & SF_PERY) != 0;
    const bool ws = (t.kind & TILE_WALLS) != 0, wn = (t.kind & TILE_WALLN) != 0;
    auto cell = [&](int x, int y) -> Pair<S> & { return box[(y - by0) * g.rs + (x - bx0)]; };
    if (sh != BOX_Y && !(px && sp.gx)) {
        const int w = 2 * HALO + tx;  // columns x0 - 3 .. x0 + tx + 2
        for (int e = id; e < w * ty; e += n) {
            const int r = e / w, x = t.x0 - HALO + (e - r * w), y = t.y0 + r;
            if (x >= 0 && x < sp.nx) continue;
            if (y >= sp.ny - (wn ? 1 : 0) || (ws && y < 1)) continue;  // no line that is used
            if (px) {
                cell(x, y) = ldv(v, i, ((x % sp.nx) + sp.nx) % sp.nx, y);
            } else if (x < 0 || x < sp.nx + HALO) {
                cell(x, y) = cell(x < 0 ? 0 : sp.nx - 1, y);
            }
        }
    }
    if (sh != BOX_X) {
        const int h = 2 * HALO + ty;
        for (int e = id; e < h * tx; e += n) {
            const int r = e / tx, x = t.x0 + (e - r * tx), y = t.y0 - HALO + r;
            if (x >= sp.nx || (y >= (ws ? 1 : 0) && y < (wn ? sp.ny - 1 : sp.ny))) continue;
            if (py) {
                cell(x, y) = ldv(v, i, x, ((y % sp.ny) + sp.ny) % sp.ny);
            } else if (y < 1) {
                cell(x, y) = ws ? extrapolate(cell(x, 1), cell(x, 2)) : cell(x, 0);
            } else if (y < sp.ny + HALO) {
                cell(x, y) = wn ? extrapolate(cell(x, sp.ny - 2), cell(x, sp.ny - 3)) : cell(x, sp.ny - 1);
            }
        }
    }
}

struct NoHook {
    template <class V>
    __device__ __forceinline__ V operator()(int, V F) const { return F; }
};

// faces of a y line at a straight wall: the wall's own face is left out (the
// wall flux is subtracted once it is known), and the faces into the wall are
// kept for its factor.  y0, s: place and direction of the line's node 0.
template <class S>
struct WallHook {
    int y0, s, ny, kind, col, tx, slot;  // slot: which of the 4 directions into the wall
    S *save;                             // [2 walls][4][tx]
    template <class V>
    __device__ __forceinline__ V operator()(int n, V F) const
    {
        const int y = y0 + s * n;
        if (kind & TILE_WALLS) {
            if (s > 0 && y == 0) F = kc<V>(0.0);
            if (s < 0 && y == 1) save[slot * tx + col] = F.x;
        }
        if (kind & TILE_WALLN) {
            if (s < 0 && y == ny - 1) F = kc<V>(0.0);
            if (s > 0 && y == ny - 2) save[(4 + slot) * tx + col] = F.x;
        }
        return F;
    }
};
// the place of direction i among the four with its sign of e_y, in the order
// of wallFluxes' sums (c_WII, c_WINV)
__device__ __forceinline__ int wall_slot_in(int i)  // c_WII[2], c_WII[3]
{
    return i == 2 || i == 4 ? 0 : i == 5 || i == 7 ? 1 : i == 6 || i == 8 ? 2 : 3;
}

// LEN flux differences of direction i along x, row `row`, columns c0 .. c0 +
// LEN - 1 of the tile, into the part array (rows of tx + 1)
template <class S, int FM, int LEN>
__device__ __forceinline__ void sweep_x(const Pair<S> *box, BoxPlace g, bool pos, int row, int c0, const FaceArg<S> &fa,
                                        Pair<S> (&out)[LEN])
{
    using V = Pair<S>;
    V v[LEN + 5];
    const V *p = box + (row + g.ry) * g.rs + c0 + g.cx;
    if constexpr (sizeof(S) == 4) {
        // two pairs per load; the line starts at an odd column of the box
        // (upwind from the left) or an even one (from the right)
        const float4 *q = reinterpret_cast<const float4 *>(p - (pos ? 4 : 2));
        float4 L[(LEN + 6) / 2];
#pragma unroll
        for (int k = 0; k < (LEN + 6) / 2; ++k) L[k] = q[k];
        if (pos) {
#pragma unroll
            for (int k = 0; k < LEN + 5; ++k)
                v[k] = (k + 1) & 1 ? make_float2(L[(k + 1) / 2].z, L[(k + 1) / 2].w) : make_float2(L[(k + 1) / 2].x, L[(k + 1) / 2].y);
            line_diffs<FM, LEN>(v, fa, out, NoHook());
        } else {
#pragma unroll
            for (int k = 0; k < LEN + 5; ++k) {
                const int j = LEN + 4 - k;
                v[k] = j & 1 ? make_float2(L[j / 2].z, L[j / 2].w) : make_float2(L[j / 2].x, L[j / 2].y);
            }
            line_diffs<FM, LEN>(v, fa, out, NoHook());
        }
    } else {
        const int s = pos ? 1 : -1;
        const V *q = pos ? p - 3 : p + LEN + 2;
#pragma unroll
        for (int k = 0; k < LEN + 5; ++k) v[k] = q[s * k];
        line_diffs<FM, LEN>(v, fa, out, NoHook());
    }
}
// node n of a line lies at column (row) c0 + n, or counted back
template <class V, int LEN>
__device__ __forceinline__ void store_line(V *part, const V (&out)[LEN], bool pos, int step, int lim)
{
#pragma unroll
    for (int n = 0; n < LEN; ++n) {
        const int k = pos ? n : LEN - 1 - n;
        if (k < lim) part[k * step] = out[n];
    }
}

template <class S, int FM, int LEN, bool HOOK>
__device__ __forceinline__ void sweep_y(const Pair<S> *box, BoxPlace g, bool pos, int col, int r0, int last, const FaceArg<S> &fa,
                                        Pair<S> (&out)[LEN], const WallHook<S> &hook)
{
    using V = Pair<S>;
    V v[LEN + 5];
    const V *p = box + col + g.cx;
    const int s = pos ? 1 : -1, r = r0 + HALO + (pos ? -3 : LEN + 2);
    if (last < 0) {  // every row of the line is in the box
        const V *q = p + r * g.rs;
        const int st = s * g.rs;
#pragma unroll
        for (int k = 0; k < LEN + 5; ++k) v[k] = q[st * k];
    } else {
#pragma unroll
        for (int k = 0; k < LEN + 5; ++k) v[k] = p[min(r + s * k, last) * g.rs];
    }
    if constexpr (HOOK) line_diffs<FM, LEN>(v, fa, out, hook);
    else line_diffs<FM, LEN>(v, fa, out, NoHook());
}

// one warp of a default tile: direction ix along x, then iy along y
// (equal for the diagonals)
template <class S, int FM>
__device__ __forceinline__ bool sweep_warp(const Tile &t, const SampleParams *gsp, const StageView<S> v, Pair<S> *sm,
                                           uint64_t *bars, int warp, int lane)
{
    using V = Pair<S>;
    constexpr FluxSmem L = flux_smem<S>(TILE_CX, TILE_CY, true, true, 12);
    constexpr int PR = TILE_CX + 1;
    const bool diag = warp >= 4;
    const int ix = diag ? warp + 1 : warp < 2 ? 1 + 2 * warp : 5 + 2 * warp;
    const int iy = diag ? warp + 1 : ix + 1;
    const bool fix = (t.kind & TILE_FIX) != 0;
    bool ok = true;
    {
        V *box = sm + box_start<S>(ix);
        const BoxPlace g = diag ? box_place<S>(BOX_XY, TILE_CX) : box_place<S>(BOX_X, TILE_CX);
        const bool pos = lat_ex(ix) > 0;
        const FaceArg<S> fa = face_arg<S>(*gsp, lat_ex(ix));
        ok = mbar_wait_bounded(&bars[ix - 1], 0, TMA_WAIT_POLLS);
        if (fix) {
            fix_box<S>(box, gsp, v, t, TILE_CX, TILE_CY, ix, lane, 32);
            __syncwarp();
        }
        const int row = lane & 7, c0 = (lane >> 3) * 8;
        V out[8];
        sweep_x<S, FM, 8>(box, g, pos, row, c0, fa, out);
        V *part = diag ? sm + L.part_off + (ix - 5) * part_pairs(TILE_CX, TILE_CY) : box;
        if (!diag) __syncwarp();
        store_line<V, 8>(part + row * PR + c0, out, pos, 1, 8);
    }
    {
        V *box = sm + box_start<S>(iy);
        const BoxPlace g = diag ? box_place<S>(BOX_XY, TILE_CX) : box_place<S>(BOX_Y, TILE_CX);
        const bool pos = lat_ey(iy) > 0;
        const FaceArg<S> fa = face_arg<S>(*gsp, lat_ey(iy));
        V out[8];
        if (!diag) {
            ok = mbar_wait_bounded(&bars[iy - 1], 0, TMA_WAIT_POLLS) && ok;
            if (fix) {
                fix_box<S>(box, gsp, v, t, TILE_CX, TILE_CY, iy, lane, 32);
                __syncwarp();
            }
        }
        if (t.kind & (TILE_WALLS | TILE_WALLN)) {
            const WallHook<S> hook{pos ? t.y0 : t.y0 + 7, pos ? 1 : -1, gsp->ny, t.kind, lane, TILE_CX, wall_slot_in(iy),
                                   reinterpret_cast<S *>(sm + L.wall_off)};
            sweep_y<S, FM, 8, true>(box, g, pos, lane, 0, -1, fa, out, hook);
        } else {
            sweep_y<S, FM, 8, false>(box, g, pos, lane, 0, -1, fa, out, WallHook<S>{});
        }
        __syncwarp();
        store_line<V, 8>(box + lane, out, pos, PR, 8);
    }
    return ok;
}

// other tile shapes: the boxes resident, in lines of 4 nodes spread over the
// block's threads
template <class S, int FM>
__device__ void sweep_block(const Tile &t, const SampleParams *gsp, const Pair<S> *slots, int slot_pairs, Pair<S> *parts,
                            S *save, int tx, int ty, int i0, int ndir, int tid, int nt)
{
    using V = Pair<S>;
    const int segx = tx / 4, segy = (ty + 3) / 4, nxi = ty * segx, per = nxi + tx * segy;
    const int PR = tx + 1, PP = part_pairs(tx, ty);
    for (int it = tid; it < ndir * per; it += nt) {
        const int d = it / per, q = it - d * per, i = i0 + d;
        const int sh = box_shape(i);
        const BoxPlace g = box_place<S>(sh, tx);
        const V *box = slots + d * slot_pairs;
        V out[4];
        if (q < nxi) {
            if (sh == BOX_Y) continue;
            const int seg = q / ty, row = q - seg * ty;
            const bool pos = lat_ex(i) > 0;
            sweep_x<S, FM, 4>(box, g, pos, row, 4 * seg, face_arg<S>(*gsp, lat_ex(i)), out);
            store_line<V, 4>(parts + part_index(i, 0) * PP + row * PR + 4 * seg, out, pos, 1, 4);
        } else {
            if (sh == BOX_X) continue;
            const int p = q - nxi, seg = p / tx, col = p - seg * tx;
            const bool pos = lat_ey(i) > 0;
            const WallHook<S> hook{pos ? t.y0 + 4 * seg : t.y0 + 4 * seg + 3, pos ? 1 : -1, gsp->ny, t.kind, col, tx,
                                   wall_slot_in(i), save};
            sweep_y<S, FM, 4, true>(box, g, pos, col, 4 * seg, box_height(sh, ty) - 1, face_arg<S>(*gsp, lat_ey(i)), out,
                                    hook);
            store_line<V, 4>(parts + part_index(i, 1) * PP + 4 * seg * PR + col, out, pos, PR, ty - 4 * seg);
        }
    }
}

// general tiles: the face of direction i along `axis` at node (x, y), solid
// nodes answering the wall flux
template <class S>
__device__ __noinline__ Pair<S> node_face(const SampleParams &sp, const StageView<S> &v, const S *alpha,
                                          const double *fref, int i, int axis, int x, int y)
{
    const int o = y * v.pitch + x;
    const uint8_t fl = v.nf[o];
    if ((fl & NF_TYPE) == 2)
        return wall_flux<S>(alpha[o], ldv(v, i, x, y), fref, i, face_arg<S>(sp, axis == 0 ? c_EX[i] : c_EY[i]));
    return flux_axis<S, S>(sp, v, x, y, i, axis, fl);
}

template <class S>
struct FluxBlocks {
    static constexpr int value = 2;
};
template <int MODE>
struct SweepBlocksF32 {
    static constexpr int value = MODE == 2 ? 3 : 2;
};

// MODE: 1 = RK3 stage 3 (fluxes of buffer 2), 2 = RK3 final (buffer 3),
// 3 = RK1 update, 4 = EULER update, 5 = EULER_EQ update (buffer 2)
// PATH: FLUX_SWEEP or FLUX_GENERAL, the tiles of one kind per launch (a
// block given the other kind returns at once).
// TC: the default tile shape, compiled in; other shapes are read from the
// arguments and give every node the same bits.
template <class S, int MODE, int PATH, bool TC>
__global__ void __launch_bounds__(256, (sizeof(S) == 4 && PATH == FLUX_SWEEP && TC) ? SweepBlocksF32<MODE>::value : 2)
k_flux(KArgs<S> a)
{
    using C = S;
    using V = Pair<S>;
    extern __shared__ __align__(128) unsigned char smem_dyn[];
    __shared__ double red[32];
    __shared__ SampleParams s_sp;  // kept out of registers: read as needed
    constexpr bool SWEEP = PATH == FLUX_SWEEP;
    const int TX = TC ? TILE_CX : a.tx, TY = TC ? TILE_CY : a.ty, NT = TX * TY;
    const int tid = threadIdx.x;
    V *sm = reinterpret_cast<V *>(smem_dyn + ((128 - (smem_u32(smem_dyn) & 127)) & 127));
    const Tile t = a.tiles[blockIdx.x];
    if (tile_sweep(t) != SWEEP) return;
    constexpr int PH = MODE == 2 ? 2 : 1;
    const SampleParams *gsp = a.samples + t.sample;
    const CUtensorMap *maps = a.tmaps + MAPS_PER_SAMPLE * t.sample + (PH == 1 ? 0 : 3);
    const S *stage = PH == 1 ? a.buf2 : a.buf3;
    const int PR = TX + 1, PP = part_pairs(TX, TY);
    constexpr FluxSmem LC = flux_smem<S>(TILE_CX, TILE_CY, true, true, 12);
    FluxSmem Lr{};
    if constexpr (!TC) Lr = flux_smem<S>(TX, TY, false, SWEEP, SWEEP ? a.slots : 0);
    const int part_off = TC ? (SWEEP ? LC.part_off : 0) : Lr.part_off;
    const int wall_off = TC ? LC.wall_off : Lr.wall_off;

    for (int k = tid; k < (int)(sizeof(SampleParams) / 4); k += NT)
        reinterpret_cast<int *>(&s_sp)[k] = reinterpret_cast<const int *>(gsp)[k];
    if constexpr (SWEEP) {
        uint64_t *bars = reinterpret_cast<uint64_t *>(sm + (TC ? LC.bar_off : Lr.bar_off));
        const int fm = tile_fm(t.kind);
        const int gx = (t.kind & TILE_GHOST) ? GHOST_X : 0;
        bool ok = true;
        if constexpr (TC) {
            const int warp = tid >> 5, lane = tid & 31;
            if (lane == 0) {
                const bool diag = warp >= 4;
                const int ix = diag ? warp + 1 : warp < 2 ? 1 + 2 * warp : 5 + 2 * warp;
                mbar_init(&bars[ix - 1], 1);
                if (!diag) mbar_init(&bars[ix], 1);
                fence_mbar_init();
                issue_box<S>(sm + box_start<S>(ix), maps, t.x0, t.y0, gx, TILE_CX, TILE_CY, ix, &bars[ix - 1]);
                if (!diag)
                    issue_box<S>(sm + box_start<S>(ix + 1), maps, t.x0, t.y0, gx, TILE_CX, TILE_CY, ix + 1, &bars[ix]);
            }
            __syncwarp();
            const StageView<S> v{stage + gsp->state_off, a.nflags + gsp->node_off, (int)gsp->plane, gsp->pitch};
            // FP64 has one form of the weights
            if (sizeof(S) == 8 ? fm != 0 : fm == 1) ok = sweep_warp<S, 1>(t, gsp, v, sm, bars, warp, lane);
            else if (fm == 2) ok = sweep_warp<S, sizeof(S) == 4 ? 2 : 1>(t, gsp, v, sm, bars, warp, lane);
            else ok = sweep_warp<S, 0>(t, gsp, v, sm, bars, warp, lane);
        } else {
            if (tid == 0) {
                for (int b = 0; b < a.slots; ++b) mbar_init(&bars[b], 1);
                fence_mbar_init();
            }
            __syncthreads();
            const StageView<S> v{stage + gsp->state_off, a.nflags + gsp->node_off, (int)gsp->plane, gsp->pitch};
            for (int i0 = 1, r = 0; i0 <= 12; i0 += a.slots, ++r) {
                const int nd = min(a.slots, 13 - i0);
                if (tid == 0) {
                    fence_proxy_async_smem();
                    for (int d = 0; d < nd; ++d)
                        issue_box<S>(sm + d * Lr.slot_pairs, maps, t.x0, t.y0, gx, TX, TY, i0 + d, &bars[d]);
                }
                // every thread waits for every copy of the round
                for (int d = 0; d < nd; ++d) ok = mbar_wait_bounded(&bars[d], r & 1, TMA_WAIT_POLLS) && ok;
                if (t.kind & TILE_FIX) {
                    for (int d = 0; d < nd; ++d) {
                        // x cells, then (they read other cells) y cells: the
                        // two touch disjoint parts of a box
                        fix_box<S>(sm + d * Lr.slot_pairs, gsp, v, t, TX, TY, i0 + d, tid, NT);
                    }
                    __syncthreads();
                }
                S *save = reinterpret_cast<S *>(sm + wall_off);
                if (sizeof(S) == 8 ? fm != 0 : fm == 1)
                    sweep_block<S, 1>(t, gsp, sm, Lr.slot_pairs, sm + part_off, save, TX, TY, i0, nd, tid, NT);
                else if (fm == 2)
                    sweep_block<S, sizeof(S) == 4 ? 2 : 1>(t, gsp, sm, Lr.slot_pairs, sm + part_off, save, TX, TY, i0, nd,
                                                           tid, NT);
                else sweep_block<S, 0>(t, gsp, sm, Lr.slot_pairs, sm + part_off, save, TX, TY, i0, nd, tid, NT);
                __syncthreads();
            }
        }
        if (!ok) atomicOr(&a.status[t.sample], STATUS_TIMEOUT);
    }
    __syncthreads();

    const SampleParams &sp = s_sp;
    const int tx = tid % TX, ty = tid / TX;
    const int x = t.x0 + tx, y = t.y0 + ty;
    const int o = y * sp.pitch + x;
    // the node's place in a part array, and the arrays' starts
    const int pn = ty * PR + tx;
    V *const parts = sm + part_off;
    auto part = [&](int i, int axis) -> V & {
        if constexpr (TC && SWEEP) {
            if (box_shape(i) == BOX_XY && axis == 0) return parts[(i - 5) * PP + pn];
            return sm[box_start<S>(i) + pn];
        } else {
            return parts[part_index(i, axis) * PP + pn];
        }
    };
    bool active = x < sp.nx && y < sp.ny;
    if (active && (!SWEEP || (t.kind & TILE_FIX))) active = (a.nflags[sp.node_off + o] & NF_TYPE) == 0;
    if (SWEEP && (t.kind & TILE_FIX) && active) {
        // at a clamped edge cFLUX's upstream face is the node's own (index
        // clamps): no difference
        const bool cx = !(sp.flags & SF_PERX), cy = !(sp.flags & SF_PERY);
#pragma unroll
        for (int i = 1; i < NQ; ++i) {
            if (cx && lat_ex(i) != 0 && x == (lat_ex(i) > 0 ? 0 : sp.nx - 1)) part(i, 0) = kc<V>(0.0);
            if (cy && lat_ey(i) != 0 && y == (lat_ey(i) > 0 ? 0 : sp.ny - 1)) part(i, 1) = kc<V>(0.0);
        }
        // straight walls: the factor of the wall node below (above), from the
        // faces into it that the sweeps kept, and its flux into this node
        const StageView<S> v{stage + sp.state_off, nullptr, (int)sp.plane, sp.pitch};
        const double *fr = a.fref + NPL * t.sample;
        const S *save = reinterpret_cast<const S *>(sm + wall_off);
        auto wall = [&](int yw, int w, const int (&in)[4], const int (&out)[4]) {
            const double dd = a.dyv[sp.yoff + yw];
            double fin = 0, fout = 0;
            V fs[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                fs[q] = ldv(v, out[q], x, yw);
                const double ci = sp.c * (lat_ey(in[q]) == 2 || lat_ey(in[q]) == -2 ? 2 : 1);
                fin = wall_in(fin, save[(4 * w + wall_slot_in(in[q])) * TX + tx], fr[in[q]], ci, dd);
                fout = wall_out(fout, (double)fs[q].x, fr[out[q]], ci, dd);
            }
            const C am1 = a.phased ? a.template alpha_as<C>()[sp.node_off + (long long)yw * sp.pitch + x]
                                   : (C)wall_ratio_m1(fin, fout);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                V &p = part(out[q], 1);
                p = xsub(p, wall_flux<C>(am1, fs[q], fr, out[q], face_arg<C>(sp, lat_ey(out[q]))));
            }
        };
        if ((t.kind & TILE_WALLS) && y == 1) wall(0, 0, {4, 7, 8, 12}, {2, 6, 5, 10});
        if ((t.kind & TILE_WALLN) && y == sp.ny - 2) wall(sp.ny - 1, 1, {2, 5, 6, 10}, {4, 8, 7, 12});
    }
    if constexpr (!SWEEP) {
        if (active) {
            const StageView<S> v{stage + sp.state_off, a.nflags + sp.node_off, (int)sp.plane, sp.pitch};
            const S *alpha = a.template alpha_as<S>() + sp.node_off;
            const double *fr = a.fref + NPL * t.sample;
#pragma unroll 1
            for (int i = 1; i < NQ; ++i)
#pragma unroll 1
                for (int axis = 0; axis < 2; ++axis) {
                    const int e = isgn(axis == 0 ? c_EX[i] : c_EY[i]);
                    if (e == 0) continue;
                    // upstream face: index(x, -e), reflected at a mirror edge
                    int m;
                    const int u = bc_index(sp, axis == 0 ? x : y, -e, axis, m);
                    const int iu = m ? (axis == 0 ? c_MIR_EW[i] : c_MIR_NS[i]) : i;
                    const V out = node_face<S>(sp, v, alpha, fr, i, axis, x, y);
                    const V in = axis == 0 ? node_face<S>(sp, v, alpha, fr, iu, 0, u, y)
                                           : node_face<S>(sp, v, alpha, fr, iu, 1, x, u);
                    parts[part_index(i, axis) * PP + pn] = xsub(out, in);
                }
        }
    }

    double res_part = 0;
    if (active) {
        V *__restrict__ st = pair_base(a.state, sp) + o;
        V *__restrict__ b3 = pair_base(a.buf3, sp) + o;
        const int PL = (int)sp.plane;
        // divergence dt (F_out - F_in)/dx of direction i (cFLUX,
        // cpuLBM.cpp:1436-1470): the parts times dt/dx and dt/dy (FP64: and |e|)
        constexpr bool F32 = sizeof(S) == 4;
        const double cs = F32 ? 1.0 : sp.c;
        const C kx = (C)__dmul_rn(a.tdx[sp.xoff + x], cs), ky = (C)__dmul_rn(a.tdy[sp.yoff + y], cs);
        auto div = [&](int i) -> V {
            const C ux = F32 || lat_ex(i) % 2 ? kx : kx + kx, uy = F32 || lat_ey(i) % 2 ? ky : ky + ky;
            const V vx = make_pair2(ux, ux), vy = make_pair2(uy, uy);
            if (i == 0) return kc<V>(0.0);
            if (box_shape(i) == BOX_X) return xmul(vx, part(i, 0));
            if (box_shape(i) == BOX_Y) return xmul(vy, part(i, 1));
            return xfma(vy, part(i, 1), xmul(vx, part(i, 0)));
        };
        constexpr bool DEV = sizeof(S) == 4;
        bool bad = false, bad_eq = false;
        MomentSums ms;       // of the new state, when the residual is wanted
        S fin_r = 0, fin_h = 0;  // NaN / Inf propagate through these sums as through FP64 ones
        if constexpr (MODE == 1) {
            // RK3 stage 3 (cpuLBM.cpp:1928-1993) and the part of the update
            // (cpuLBM.cpp:1999-2042) that does not need the stage-3 fluxes
            const int gd = ghost_offset(sp, x);
            V fv[NQ];
#pragma unroll
            for (int i = 0; i < NQ; ++i) fv[i] = st[i * PL];
            // stage-1 moments (= stage 2's) and the moments of f - div F(f2)
            // (macroProp3, cpuLBM.cpp:973-1032)
            MomentSums s1, s3;
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                const double f = (double)fv[i].x, h = (double)fv[i].y;
                s1.add(i, f, h);
                const V D = div(i);
                s3.add(i, i ? __dsub_rn(f, (double)D.x) : f, i ? __dsub_rn(h, (double)D.y) : h);
            }
            const Macro m1 = s1.macro(sp), m3 = s3.macro(sp);
            const EqArgs<C, DEV> q1(m1.rho, m1.ux, m1.uy, m1.T, sp);
            const EqArgs<C, DEV> q3(m3.rho, m3.ux, m3.uy, m3.T, sp);
            const Stage3<C> s(m1, m3, sp);
            double sf3 = 0;
            auto family = [&](const int fam) {
                C e1f[4], e1h[4], e3f[4], e3h[4];
                q1.fam(fam, e1f, e1h);
                q3.fam(fam, e3f, e3h);
                const int i0 = fam == 0 ? 0 : 4 * fam - 3, n = fam == 0 ? 1 : 4;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (k >= n) break;
                    const int i = i0 + k;
                    sf3 += (double)e3f[k];
                    V n3, acc;
                    s.update(i, fv[i], div(i), make_pair2(e1f[k], e1h[k]), make_pair2(e3f[k], e3h[k]), n3, acc);
                    b3[i * PL] = n3;
                    if (gd) b3[i * PL + gd] = n3;
                    st[i * PL] = acc;
                }
            };
#pragma unroll
            for (int fam = 0; fam < 4; ++fam) family(fam);
            bad_eq = fabs(sf3 - (m3.rho - sp.rho0)) > a.eq_tol * (sizeof(C) == 8 ? 1.0 : fmax(1.0, fabs(m3.rho)));
        } else if constexpr (MODE == 2) {
            // final RK3 combination (cpuLBM.cpp:1999-2042): f = acc - D3/2
            V acc[NQ];
#pragma unroll
            for (int i = 0; i < NQ; ++i) acc[i] = st[i * PL];
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                const V n = i ? xfma(kc<V>(-0.5), div(i), acc[i]) : acc[i];
                st[i * PL] = n;
                fin_r += n.x;
                fin_h += n.y;
                if (a.want_residual) ms.add(i, (double)n.x, (double)n.y);
            }
        } else {
            // RK1 update (cpuLBM.cpp:1674-1710), EULER (:2130-2168), EULER_EQ (:2220-2258)
            V fv[NQ];
#pragma unroll
            for (int i = 0; i < NQ; ++i) fv[i] = st[i * PL];
            const Macro m = node_macro_rd([&](int i) { return fv[i]; }, sp);
            const EqArgs<C, DEV> q(m.rho, m.ux, m.uy, m.T, sp);
            const Update<C, MODE> u(m, sp);
            double sf = 0;
            auto family = [&](const int fam) {
                C fe[4], he[4];
                q.fam(fam, fe, he);
                const int i0 = fam == 0 ? 0 : 4 * fam - 3, n = fam == 0 ? 1 : 4;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (k >= n) break;
                    const int i = i0 + k;
                    sf += (double)fe[k];
                    const V nv = u.value(i, fv[i], div(i), make_pair2(fe[k], he[k]));
                    st[i * PL] = nv;
                    fin_r += nv.x;
                    fin_h += nv.y;
                    if (a.want_residual) ms.add(i, (double)nv.x, (double)nv.y);
                }
            };
#pragma unroll
            for (int fam = 0; fam < 4; ++fam) family(fam);
            if (MODE >= 4)
                bad_eq = fabs(sf - (m.rho - sp.rho0)) > a.eq_tol * (sizeof(C) == 8 ? 1.0 : fmax(1.0, fabs(m.rho)));
        }
        if (MODE != 1) {
            if (a.want_residual) {
                // macroPropShort of the new state: the residual's T, and the
                // finiteness / positive-density check
                const Macro mn = ms.macro(sp);
                bad = !(mn.rho > 0.0) || !isfinite(mn.rho) || !isfinite(mn.T) || !isfinite(mn.ux) || !isfinite(mn.uy);
                const double d = mn.T - a.told[sp.node_off + o];
                res_part = d * d;
            } else {
                const double r = (double)fin_r + sp.rho0;
                bad = !(r > 0.0) || !isfinite(r) || !isfinite((double)fin_h);
            }
        }
        if (bad_eq) atomicOr(&a.status[t.sample], STATUS_EQ);
        if (bad) atomicOr(&a.status[t.sample], STATUS_NONFINITE);
    }
    if (a.want_residual && MODE != 1) {
        // per-tile partial sum, fixed order (deterministic)
        for (int off = 16; off > 0; off >>= 1) res_part += __shfl_down_sync(0xffffffffu, res_part, off);
        if ((tid & 31) == 0) red[tid >> 5] = res_part;
        __syncthreads();
        if (tid == 0) {
            double s = 0;
            for (int w = 0; w < (NT + 31) / 32; ++w) s += red[w];
            a.partial[t.gid] = s;
        }
    }
}

// ----------------------------------------------------------------- launchers
template <class S, int PATH, bool TC>
void launch_flux_t(int mode, const KArgs<S> &k, int ntiles, int NT, size_t sm, cudaStream_t st)
{
    switch (mode) {
    case 1: k_flux<S, 1, PATH, TC><<<ntiles, NT, sm, st>>>(k); break;
    case 2: k_flux<S, 2, PATH, TC><<<ntiles, NT, sm, st>>>(k); break;
    case 3: k_flux<S, 3, PATH, TC><<<ntiles, NT, sm, st>>>(k); break;
    case 4: k_flux<S, 4, PATH, TC><<<ntiles, NT, sm, st>>>(k); break;
    default: k_flux<S, 5, PATH, TC><<<ntiles, NT, sm, st>>>(k); break;
    }
}

template <class S>
cudaError_t launch_flux(int mode, const KArgs<S> &a, int ntiles, int path, cudaStream_t st)
{
    KArgs<S> k = a;
    const bool def = k.tx == TILE_CX && k.ty == TILE_CY, sweep = path == FLUX_SWEEP;
    k.slots = def ? 12 : flux_slots<S>(k.tx, k.ty);
    const int NT = k.tx * k.ty;
    const size_t sm = flux_smem_bytes_t<S>(k.tx, k.ty, sweep);
    if (sweep) {
        if (def) launch_flux_t<S, FLUX_SWEEP, true>(mode, k, ntiles, NT, sm, st);
        else launch_flux_t<S, FLUX_SWEEP, false>(mode, k, ntiles, NT, sm, st);
    } else {
        launch_flux_t<S, FLUX_GENERAL, false>(mode, k, ntiles, NT, sm, st);
    }
    return cudaGetLastError();
}

template <class S>
cudaError_t prepare_flux()
{
    const int maxsm = 224 * 1024;
    cudaError_t e = cudaSuccess;
#define UQ_FLUX_SMEM1(M, P, T)                                                                             \
    if (e == cudaSuccess)                                                                                  \
        e = cudaFuncSetAttribute(k_flux<S, M, P, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxsm);
#define UQ_FLUX_SMEM(M) \
    UQ_FLUX_SMEM1(M, FLUX_SWEEP, true) UQ_FLUX_SMEM1(M, FLUX_SWEEP, false) UQ_FLUX_SMEM1(M, FLUX_GENERAL, false)
    UQ_FLUX_SMEM(1) UQ_FLUX_SMEM(2) UQ_FLUX_SMEM(3) UQ_FLUX_SMEM(4) UQ_FLUX_SMEM(5)
#undef UQ_FLUX_SMEM
#undef UQ_FLUX_SMEM1
    return e;
}

}  // namespace uqlbm
