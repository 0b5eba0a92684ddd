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
#pragma once

#include "lbm_box.h"
#include "lbm_node.cuh"
#include "tma.cuh"

#include <cuda_runtime.h>

#include <type_traits>

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
// boxes are still being swept along y).  Other tile shapes: `slots` boxes at a time
// and all 16 parts apart.  General tiles: the parts only.
struct FluxSmem {
    int slots;       // boxes resident at a time
    int slot_pairs;  // pairs per slot (not the default tile)
    int part_off;    // the parts (default tile: the diagonals' x parts), in pairs
    int wall_off;    // saved wall faces (general tiles: faces into the tile), in pairs
    int bar_off;     // mbarriers, in pairs
    size_t bytes;    // with 128 bytes of base-alignment slack
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
    // [2 walls][4][tx] values of S; general tiles: the faces into the tile
    off += sweep ? (4 * tx + 15) / 16 * 16 : 8 * (tx + ty);
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
__device__ __noinline__ void fix_box(Pair<S> *box, const SampleParams &sp, const S *stage, const Tile t, int tx, int ty,
                                     int i, int id, int n)
{
    const StageView<S> v{stage + sp.state_off, nullptr, (int)sp.plane, sp.pitch};
    const int sh = box_shape(i);
    const BoxPlace g = box_place<S>(sh, tx);
    const int bx0 = t.x0 - g.cx, by0 = t.y0 - g.ry;  // domain place of the box's first cell
    const bool px = (sp.flags & SF_PERX) != 0, py = (sp.flags & SF_PERY) != 0;
    const bool ws = (t.kind & TILE_WALLS) != 0, wn = (t.kind & TILE_WALLN) != 0;
    auto cell = [&](int x, int y) -> Pair<S> & { return box[(y - by0) * g.rs + (x - bx0)]; };
    if (sh != BOX_Y && !(px && sp.gx)) {
        // the columns left of 0 and from nx on that a node of the tile sees
        const int left = max(HALO - t.x0, 0), right = min(max(t.x0 + tx + HALO - sp.nx, 0), HALO);
        for (int e = id; e < (left + right) * ty; e += n) {
            const int c = e / ty, y = t.y0 + (e - c * ty), x = c < left ? t.x0 - HALO + c : sp.nx + (c - left);
            if (y >= sp.ny - (wn ? 1 : 0) || (ws && y < 1)) continue;  // no line that is used
            cell(x, y) = px ? ldv(v, i, ((x % sp.nx) + sp.nx) % sp.nx, y) : cell(x < 0 ? 0 : sp.nx - 1, y);
        }
    }
    if (sh != BOX_X) {
        // the rows before `first` and from `last` on that a node of the tile
        // sees; a wall row counts as outside
        const int first = min(t.y0 + ty + HALO, ws ? 1 : 0), last = max(t.y0 - HALO, wn ? sp.ny - 1 : sp.ny);
        const int end = min(t.y0 + ty, sp.ny) + HALO;
        for (int col = id; col < tx; col += n) {
            const int x = t.x0 + col;
            if (x >= sp.nx) continue;
            for (int y = t.y0 - HALO; y < first; ++y)
                cell(x, y) = py ? ldv(v, i, x, ((y % sp.ny) + sp.ny) % sp.ny)
                           : ws ? extrapolate(cell(x, 1), cell(x, 2)) : cell(x, 0);
            for (int y = last; y < end; ++y)
                cell(x, y) = py ? ldv(v, i, x, ((y % sp.ny) + sp.ny) % sp.ny)
                           : wn ? extrapolate(cell(x, sp.ny - 2), cell(x, sp.ny - 3)) : cell(x, sp.ny - 1);
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
// node n of a line lies at column (row) n of its segment, or counted back;
// both written out, so that every address is a constant distance from one
template <class V, int LEN>
__device__ __forceinline__ void store_line(V *part, const V (&out)[LEN], bool pos, int step)
{
    if (pos) {
#pragma unroll
        for (int n = 0; n < LEN; ++n) part[n * step] = out[n];
    } else {
#pragma unroll
        for (int n = 0; n < LEN; ++n) part[(LEN - 1 - n) * step] = out[n];
    }
}
// the same of a line that may reach beyond the tile (other tile shapes)
template <class V, int LEN>
__device__ __forceinline__ void store_line_to(V *part, const V (&out)[LEN], bool pos, int step, int lim)
{
#pragma unroll
    for (int n = 0; n < LEN; ++n) {
        const int k = pos ? n : LEN - 1 - n;
        if (k < lim) part[k * step] = out[n];
    }
}

// the same along y, column `col`, rows r0 .. r0 + LEN - 1.  last: the last row
// of the box, where a line may reach beyond it (LAST, other tile shapes)
template <class S, int FM, int LEN, bool HOOK, bool LAST>
__device__ __forceinline__ void sweep_y(const Pair<S> *box, BoxPlace g, bool pos, int col, int r0, int last,
                                        const FaceArg<S> &fa, Pair<S> (&out)[LEN], const WallHook<S> &hook)
{
    using V = Pair<S>;
    V v[LEN + 5];
    const V *p = box + col + g.cx;
    if constexpr (LAST) {
        const int s = pos ? 1 : -1, r = r0 + HALO + (pos ? -3 : LEN + 2);
#pragma unroll
        for (int k = 0; k < LEN + 5; ++k) v[k] = p[min(r + s * k, last) * g.rs];
    } else {
        const V *q = p + r0 * g.rs;
        if (pos) {
#pragma unroll
            for (int k = 0; k < LEN + 5; ++k) v[k] = q[k * g.rs];
        } else {
#pragma unroll
            for (int k = 0; k < LEN + 5; ++k) v[k] = q[(LEN + 5 - k) * g.rs];
        }
    }
    if constexpr (HOOK) line_diffs<FM, LEN>(v, fa, out, hook);
    else line_diffs<FM, LEN>(v, fa, out, NoHook());
}

// one warp of a default tile: direction ix along x, then iy along y
// (equal for the diagonals)
template <class S, int FM>
__device__ __forceinline__ bool sweep_warp(const Tile &t, const SampleParams &sp, const S *stage, Pair<S> *sm, S *save,
                                           uint64_t *bars, int warp, int lane)
{
    using V = Pair<S>;
    constexpr FluxSmem L = flux_smem<S>(TILE_CX, TILE_CY, true, true, 12);
    constexpr int PR = TILE_CX + 1, PP = part_pairs(TILE_CX, TILE_CY);
    const bool diag = warp >= 4;
    const int ix = diag ? warp + 1 : warp < 2 ? 1 + 2 * warp : 5 + 2 * warp;
    const int iy = diag ? warp + 1 : ix + 1;
    const bool fix = (t.kind & TILE_FIX) != 0;
    bool ok = true;
    {
        V *box = sm + box_start<S>(ix);
        const BoxPlace g = diag ? box_place<S>(BOX_XY, TILE_CX) : box_place<S>(BOX_X, TILE_CX);
        const bool pos = lat_ex(ix) > 0;
        const FaceArg<S> fa = face_arg<S>(t.c, t.eps1, lat_ex(ix));
        ok = mbar_wait_bounded(&bars[ix - 1], 0, TMA_WAIT_POLLS);
        if (fix) {
            fix_box<S>(box, sp, stage, t, TILE_CX, TILE_CY, ix, lane, 32);
            __syncwarp();
        }
        const int row = lane & 7, c0 = (lane >> 3) * 8;
        V out[8];
        sweep_x<S, FM, 8>(box, g, pos, row, c0, fa, out);
        V *part = diag ? sm + L.part_off + (ix - 5) * PP : box;
        if (!diag) __syncwarp();
        store_line<V, 8>(part + row * PR + c0, out, pos, 1);
    }
    {
        V *box = sm + box_start<S>(iy);
        const bool pos = lat_ey(iy) > 0;
        const FaceArg<S> fa = face_arg<S>(t.c, t.eps1, lat_ey(iy));
        V out[8];
        if (!diag) {
            ok = mbar_wait_bounded(&bars[iy - 1], 0, TMA_WAIT_POLLS) && ok;
            if (fix) {
                fix_box<S>(box, sp, stage, t, TILE_CX, TILE_CY, iy, lane, 32);
                __syncwarp();
            }
        }
        const bool walls = (t.kind & (TILE_WALLS | TILE_WALLN)) != 0;
        const WallHook<S> hook{pos ? t.y0 : t.y0 + 7, pos ? 1 : -1, walls ? sp.ny : 0, t.kind, lane, TILE_CX,
                               wall_slot_in(iy), save};
        // (one copy of the sweep for both box widths)
        const BoxPlace g = diag ? box_place<S>(BOX_XY, TILE_CX) : box_place<S>(BOX_Y, TILE_CX);
        if (walls) sweep_y<S, FM, 8, true, false>(box, g, pos, lane, 0, 0, fa, out, hook);
        else sweep_y<S, FM, 8, false, false>(box, g, pos, lane, 0, 0, fa, out, hook);
        __syncwarp();
        store_line<V, 8>(box + lane, out, pos, PR);
    }
    return ok;
}

// other tile shapes: the boxes resident, in lines of 4 nodes spread over the
// block's threads
template <class S, int FM>
__device__ void sweep_block(const Tile &t, const SampleParams &sp, const Pair<S> *slots, int slot_pairs, Pair<S> *parts,
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
            sweep_x<S, FM, 4>(box, g, pos, row, 4 * seg, face_arg<S>(t.c, t.eps1, lat_ex(i)), out);
            store_line_to<V, 4>(parts + part_index(i, 0) * PP + row * PR + 4 * seg, out, pos, 1, 4);
        } else {
            if (sh == BOX_X) continue;
            const int p = q - nxi, seg = p / tx, col = p - seg * tx;
            const bool pos = lat_ey(i) > 0;
            const WallHook<S> hook{pos ? t.y0 + 4 * seg : t.y0 + 4 * seg + 3, pos ? 1 : -1, sp.ny, t.kind, col, tx,
                                   wall_slot_in(i), save};
            sweep_y<S, FM, 4, true, true>(box, g, pos, col, 4 * seg, box_height(sh, ty) - 1, face_arg<S>(t.c, t.eps1, lat_ey(i)), out,
                                    hook);
            store_line_to<V, 4>(parts + part_index(i, 1) * PP + 4 * seg * PR + col, out, pos, PR, ty - 4 * seg);
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

// the a-th direction (0..7) that moves along an axis
__host__ __device__ constexpr int moving(int a, int axis) { return a < 2 ? 1 + 2 * a + axis : a < 6 ? a + 3 : 2 * a - 3 + axis; }

// General tiles: every face once.  Each thread answers the faces of its own
// node; those that enter the tile from outside (the upstream node wrapped,
// clamped or, at a mirror edge, of the reflected direction) are shared out
// over the block's threads.  The faces' arithmetic bounds these tiles, not
// memory: a 1024^2 step with 64 obstacles took 0.770 ms (FP64 1.051) with two
// faces per node, axis and direction, 0.621 (0.860) with one.
template <class S>
__device__ __forceinline__ void face_parts(const Tile &t, const SampleParams &sp, const StageView<S> &v, const S *alpha,
                                           const double *fref, Pair<S> *parts, Pair<S> *edges, int TX, int TY, int tid,
                                           int NT)
{
    using V = Pair<S>;
    const int PR = TX + 1, PP = part_pairs(TX, TY), tx = tid % TX, ty = tid / TX, pn = ty * PR + tx;
    const int x = t.x0 + tx, y = t.y0 + ty, xe = min(t.x0 + TX, sp.nx), ye = min(t.y0 + TY, sp.ny);
    const bool in = x < xe && y < ye;
    if (in) {
#pragma unroll 1
        for (int k = 0; k < 16; ++k) {
            const int axis = k >> 3, i = moving(k & 7, axis);
            parts[part_index(i, axis) * PP + pn] = node_face<S>(sp, v, alpha, fref, i, axis, x, y);
        }
    }
#pragma unroll 1
    for (int k = tid; k < 8 * (TX + TY); k += NT) {
        const int axis = k >= 8 * TY, r = axis ? k - 8 * TY : k, n = axis ? TX : TY;
        const int i = moving(r / n, axis), e = axis ? c_EY[i] : c_EX[i], j = r % n;
        // the tile's first node downstream of the face
        const int fx = axis ? t.x0 + j : e > 0 ? t.x0 : xe - 1, fy = axis ? (e > 0 ? t.y0 : ye - 1) : t.y0 + j;
        if (fx >= xe || fy >= ye || (v.nf[fy * v.pitch + fx] & NF_TYPE) != 0) continue;
        int m;
        const int u = bc_index(sp, axis ? fy : fx, e > 0 ? -1 : 1, axis, m);
        const int iu = m ? (axis ? c_MIR_NS[i] : c_MIR_EW[i]) : i;
        edges[k] = node_face<S>(sp, v, alpha, fref, iu, axis, axis ? fx : u, axis ? u : fy);
    }
    __syncthreads();
#pragma unroll
    for (int axis = 0; axis < 2; ++axis) {
        V d[8];
        if (in) {
#pragma unroll
            for (int a = 0; a < 8; ++a) {
                const int i = moving(a, axis), up = (axis ? lat_ey(i) : lat_ex(i)) > 0 ? -1 : 1;
                const int first = axis ? (up < 0 ? t.y0 : ye - 1) : up < 0 ? t.x0 : xe - 1;
                const V *p = parts + part_index(i, axis) * PP + pn;
                const V *q = (axis ? y : x) != first ? p + up * (axis ? PR : 1)
                                                     : edges + (axis ? 8 * TY + a * TX + tx : a * TY + ty);
                d[a] = xsub(*p, *q);
            }
        }
        __syncthreads();
        if (in) {
#pragma unroll
            for (int a = 0; a < 8; ++a) parts[part_index(moving(a, axis), axis) * PP + pn] = d[a];
        }
    }
}

// the whole block of a default tile: each warp its directions
template <class S>
__device__ __forceinline__ bool sweep_tile(const Tile &t, const SampleParams &sp, const S *stage, Pair<S> *sm, S *save,
                                           uint64_t *bars, int warp, int lane)
{
    const int fm = tile_fm(t.kind);
    // FP64 has one form of the weights
    if (sizeof(S) == 8 ? fm != 0 : fm == 1) return sweep_warp<S, 1>(t, sp, stage, sm, save, bars, warp, lane);
    if (fm == 2) return sweep_warp<S, sizeof(S) == 4 ? 2 : 1>(t, sp, stage, sm, save, bars, warp, lane);
    return sweep_warp<S, 0>(t, sp, stage, sm, save, bars, warp, lane);
}

// a warp's lane 0 asks for the boxes of the warp's directions (maps: the stage
// buffer's three)
template <class S>
__device__ __forceinline__ void issue_warp(const Tile &t, const CUtensorMap *maps, Pair<S> *sm, uint64_t *bars, int warp)
{
    const bool diag = warp >= 4;
    const int ix = diag ? warp + 1 : warp < 2 ? 1 + 2 * warp : 5 + 2 * warp;
    const int gx = (t.kind & TILE_GHOST) ? GHOST_X : 0;
    issue_box<S>(sm + box_start<S>(ix), maps, t.x0, t.y0, gx, TILE_CX, TILE_CY, ix, &bars[ix - 1]);
    if (!diag) issue_box<S>(sm + box_start<S>(ix + 1), maps, t.x0, t.y0, gx, TILE_CX, TILE_CY, ix + 1, &bars[ix]);
}

// a node's flux differences in shared memory.  OVER: the default tile's, over
// the boxes (sm: the tile's copy); else in the 16 part arrays (sm: the first)
template <class S, bool OVER>
struct NodeParts {
    Pair<S> *sm;
    int pn, PP;  // the node's place in an array; pairs per array
    __device__ __forceinline__ Pair<S> &operator()(int i, int axis) const
    {
        if constexpr (OVER) {
            constexpr FluxSmem L = flux_smem<S>(TILE_CX, TILE_CY, true, true, 12);
            if (box_shape(i) == BOX_XY && axis == 0)
                return sm[L.part_off + (i - 5) * part_pairs(TILE_CX, TILE_CY) + pn];
            return sm[box_start<S>(i) + pn];
        } else {
            return sm[part_index(i, axis) * PP + pn];
        }
    }
};

// Whether the per-node half loads the state before the block's barrier: the
// loads then run while other warps sweep.  FP64 (3 % of a step, and flux_free
// needs it) and RK1, which has registers for it; FP32 RK3 spills instead
// (1.32 -> 1.36 ms per step of a 64-sample ensemble).
template <class S>
__host__ __device__ constexpr bool flux_early(int mode)
{
    return sizeof(S) == 8 || mode == 3;
}

// FP64, ahead of the block's barrier: everything that needs no flux (a 1024^2
// step 0.471 -> 0.449 ms against forming it after the barrier).  v is the
// state, and becomes the new value but for its flux term (RK3 stage 3: what
// stage 3 relaxes from); m: the state's moment sums.  Whether the
// equilibrium's mass check fails.
template <int MODE, bool LAW>
__device__ __forceinline__ bool flux_free(double2 (&v)[NQ], MomentSums &ms, const SampleParams &sp, double eq_tol)
{
#pragma unroll
    for (int i = 0; i < NQ; ++i) ms.add(i, v[i].x, v[i].y);
    const Macro m = ms.macro<LAW>(sp);
    EqArgs<double, false> q(m.rho, m.ux, m.uy, m.T, sp);
    const std::conditional_t<MODE == 1, Stage3Base, Update<double, MODE>> u(m, sp);
    double sf = 0;
#pragma unroll
    for (int fam = 0; fam < 4; ++fam) {
        double fe[4], he[4];
        q.part();
        q.fam(fam, fe, he);
#pragma unroll
        for (int k = 0; k < (fam ? 4 : 1); ++k) {
            const int i = fam ? 4 * fam - 3 + k : 0;
            sf += fe[k];
            v[i] = u.base(i, v[i], make_double2(fe[k], he[k]));
        }
    }
    return MODE >= 4 && fabs(sf - m.rho) > eq_tol;
}

// The per-node half of a stencil phase (MODE as k_flux): the node's
// divergences from its parts, then the RK3 stage 3 or the update.  The
// block's barrier between the sweeps and this lies inside, after the loads
// that do not depend on the sweeps.
template <class S, int MODE, bool SWEEP, bool LAW, bool NEXT, class PART>
__device__ __forceinline__ void node_phase(const KArgs<S> &a, const Tile &t, const SampleParams &sp, const PART &part,
                                           const S *save, double *red, int TX, int NT, int tid)
{
    using C = S;
    using V = Pair<S>;
    constexpr bool F32 = sizeof(S) == 4, DEV = F32;
    constexpr bool EARLY = flux_early<S>(MODE);
    if (!EARLY) __syncthreads();
    const int tx = tid % TX, ty = tid / TX;
    const int x = t.x0 + tx, y = t.y0 + ty;
    const int o = y * sp.pitch + x, PL = (int)sp.plane;
    bool active = x < sp.nx && y < sp.ny;
    if (active && (!SWEEP || (t.kind & TILE_FIX))) active = (a.nflags[sp.node_off + o] & NF_TYPE) == 0;
    V *__restrict__ st = pair_base(a.state, sp) + o;
    C kx, ky;  // dt/dx, dt/dy (FP64: times |e|)
    V fv[NQ];  // the state (after RK3 stage 3: the update's partial sum)
    bool bad = false, bad_eq = false;
    MomentSums m0;  // FP64: the state's moment sums
    auto load = [&]() {
        const double cs = F32 ? 1.0 : sp.c;
        kx = (C)__dmul_rn(a.tdx[sp.xoff + x], cs);
        ky = (C)__dmul_rn(a.tdy[sp.yoff + y], cs);
        if (EARLY || MODE != 1) {
#pragma unroll
            for (int i = 0; i < NQ; ++i) fv[i] = st[i * PL];
        }
    };
    if (EARLY) {
        if (active) {
            load();
            if constexpr (!F32 && MODE != 2) bad_eq = flux_free<MODE, LAW>(fv, m0, sp, a.eq_tol);
        }
        __syncthreads();
    }
    pdl_trigger();
    double res_part = 0;
    if (active) {
        const S *stage = MODE == 2 ? a.buf3 : a.buf2;
        if (SWEEP && (t.kind & TILE_FIX)) {
            // at a clamped edge cFLUX's upstream face is the node's own (index
            // clamps): no difference
            const bool cx = !(sp.flags & SF_PERX), cy = !(sp.flags & SF_PERY);
#pragma unroll
            for (int i = 1; i < NQ; ++i) {
                if (cx && lat_ex(i) != 0 && x == (lat_ex(i) > 0 ? 0 : sp.nx - 1)) part(i, 0) = kc<V>(0.0);
                if (cy && lat_ey(i) != 0 && y == (lat_ey(i) > 0 ? 0 : sp.ny - 1)) part(i, 1) = kc<V>(0.0);
            }
            // straight walls: the factor of the wall node below (above), from
            // the faces into it that the sweeps kept, and its flux into this node
            const StageView<S> v{stage + sp.state_off, nullptr, (int)sp.plane, sp.pitch};
            const double *fr = a.fref + NPL * t.sample;
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
        if (!EARLY) load();
        // divergence dt (F_out - F_in)/dx of direction i (cFLUX,
        // cpuLBM.cpp:1436-1470): the parts times dt/dx and dt/dy (FP64: and |e|)
        auto div = [&](int i) -> V {
            const C ux = F32 || lat_ex(i) % 2 ? kx : kx + kx, uy = F32 || lat_ey(i) % 2 ? ky : ky + ky;
            const V vx = make_pair2(ux, ux), vy = make_pair2(uy, uy);
            if (i == 0) return kc<V>(0.0);
            if (box_shape(i) == BOX_X) return xmul(vx, part(i, 0));
            if (box_shape(i) == BOX_Y) return xmul(vy, part(i, 1));
            return xfma(vy, part(i, 1), xmul(vx, part(i, 0)));
        };
        MomentSums ms;           // of the new state, when the residual is wanted
        S fin_r = 0, fin_h = 0;  // NaN / Inf propagate through these sums as through FP64 ones
        if constexpr (MODE == 1 && !F32) {
            // RK3 stage 3 and the part of the update that does not need the
            // stage-3 fluxes, from the moments of f - div F(f2)
            V *__restrict__ b3 = pair_base(a.buf3, sp) + o;
            MomentSums md;
#pragma unroll
            for (int i = 1; i < NQ; ++i) {
                const V D = div(i);
                md.add(i, D.x, D.y);
            }
            const Macro m3 = m0.less(md).template macro<LAW>(sp);
            EqArgs<C, DEV> q3(m3.rho, m3.ux, m3.uy, m3.T, sp);
            const Stage3Rest s(m3, sp);
            double sf3 = 0;
#pragma unroll
            for (int fam = 0; fam < 4; ++fam) {
                C ef[4], eh[4];
                asm volatile("" ::: "memory");  // (and the flux differences are read again)
                q3.part();
                q3.fam(fam, ef, eh);
#pragma unroll
                for (int k = 0; k < (fam ? 4 : 1); ++k) {
                    const int i = fam ? 4 * fam - 3 + k : 0;
                    sf3 += ef[k];
                    V n3, acc;
                    s.update(i, fv[i], div(i), make_pair2(ef[k], eh[k]), n3, acc);
                    b3[i * PL] = n3;
                    st[i * PL] = acc;
                }
            }
            if (const int gd = ghost_offset(sp, x)) {
#pragma unroll 1
                for (int i = 0; i < NQ; ++i) b3[i * PL + gd] = b3[i * PL];
            }
            bad_eq = fabs(sf3 - m3.rho) > a.eq_tol;
        } else if constexpr (MODE == 1) {
            // RK3 stage 3 (cpuLBM.cpp:1928-1993) and the part of the update
            // (cpuLBM.cpp:1999-2042) that does not need the stage-3 fluxes
            const V *__restrict__ b2 = pair_base(a.buf2, sp) + o;
            V *__restrict__ b3 = pair_base(a.buf3, sp) + o;
            // stage-1 moments (= stage 2's) and the moments of f - div F(f2)
            // (macroProp3, cpuLBM.cpp:973-1032)
            MomentSums s1, s3;
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                const V v = st[i * PL];
                const double f = (double)v.x, h = (double)v.y;
                s1.add(i, f, h);
                const V D = div(i);
                s3.add(i, i ? __dsub_rn(f, (double)D.x) : f, i ? __dsub_rn(h, (double)D.y) : h);
            }
            const Macro m1 = s1.template macro<LAW>(sp), m3 = s3.template macro<LAW>(sp);
            const EqArgs<C, DEV> q1(m1.rho, m1.ux, m1.uy, m1.T, sp);
            const EqArgs<C, DEV> q3(m3.rho, m3.ux, m3.uy, m3.T, sp);
            const Stage3 s(m1, m3, sp);
            double sf3 = 0;
            // family by family; the state is loaded a second time rather than
            // kept (13 pairs of registers, better used for the loads ahead)
            V gv[4], g2[4];
            auto fetch = [&](const int fam) {
                const int i0 = fam == 0 ? 0 : 4 * fam - 3, n = fam == 0 ? 1 : 4;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k < n) {
                        gv[k] = load_again(st + (i0 + k) * PL);
                        g2[k] = b2[(i0 + k) * PL];
                    }
            };
            auto family = [&](const int fam) {
                const int i0 = fam == 0 ? 0 : 4 * fam - 3, n = fam == 0 ? 1 : 4;
                V hv[4], d2[4];
                fetch(fam);
                {
                    C ef[4], eh[4];
                    q1.fam(fam, ef, eh);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (k < n) {
                            hv[k] = gv[k];
                            d2[k] = xsub(make_pair2(ef[k], eh[k]), g2[k]);
                        }
                }
                C ef[4], eh[4];
                q3.fam(fam, ef, eh);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (k >= n) break;
                    const int i = i0 + k;
                    sf3 += (double)ef[k];
                    V n3, acc;
                    s.update(i, hv[k], div(i), d2[k], make_pair2(ef[k], eh[k]), n3, acc);
                    b3[i * PL] = n3;
                    st[i * PL] = acc;
                }
            };
#pragma unroll
            for (int fam = 0; fam < 4; ++fam) family(fam);
            // the images of nodes near a periodic edge, read back by the few
            // threads that have one (a store in the loop above would cost
            // every thread its predicate)
            if (const int gd = ghost_offset(sp, x)) {
#pragma unroll 1
                for (int i = 0; i < NQ; ++i) b3[i * PL + gd] = b3[i * PL];
            }
            bad_eq = fabs(sf3 - (m3.rho - sp.rho0)) > a.eq_tol * (sizeof(C) == 8 ? 1.0 : fmax(1.0, fabs(m3.rho)));
        } else if constexpr (MODE == 2 || !F32) {
            // final RK3 combination (cpuLBM.cpp:1999-2042): f = acc - D3/2;
            // the other updates' flux term
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                V n = fv[i];
                if (i) n = MODE == 2 ? xfma(kc<V>(-0.5), div(i), n) : xsub(n, div(i));
                if (i || MODE != 2) st[i * PL] = n;
                if (NEXT) fv[i] = n;
                fin_r += n.x;
                fin_h += n.y;
                if (NEXT || a.want_residual) ms.add(i, (double)n.x, (double)n.y);
            }
        } else {
            // RK1 update (cpuLBM.cpp:1674-1710), EULER (:2130-2168), EULER_EQ (:2220-2258)
            const Macro m = node_macro_rd<LAW>([&](int i) { return fv[i]; }, sp);
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
        if constexpr (NEXT) {
            // the next step's stages 1 and 2, into the buffer that this
            // phase does not read
            V *__restrict__ b2 = pair_base(a.buf2, sp) + o;
            bad_eq = first_stage<S, 1>(fv, ms.template macro<LAW>(sp), sp, a.eq_tol, [&](int i, V nv) { b2[i * PL] = nv; });
            if (const int gd = ghost_offset(sp, x)) {
#pragma unroll 1
                for (int i = 0; i < NQ; ++i) b2[i * PL + gd] = b2[i * PL];
            }
        }
        if (MODE != 1) {
            if (!NEXT && a.want_residual) {
                // macroPropShort of the new state: the residual's T, and the
                // finiteness / positive-density check
                const Macro mn = ms.template macro<false>(sp);  // (no relaxation time)
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
    if (!NEXT && a.want_residual && MODE != 1) {
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

// Blocks per SM.  FP32 RK3 stage 3 takes 128 registers and two blocks: at three
// (160 bytes of spills) the kernel alone is 4 % faster, but a 64-sample
// ensemble's step goes from 1.32 to 1.34 ms, the board being at its power
// limit.  The other FP32 phases fit 80 registers and three blocks (the final
// phase with the next step's stages 1.29 ms per step; at two 1.37; four
// without them +1 %).  FP64 has no room for a third block's registers.
template <class S, int MODE, bool SWEEP>
struct FluxBlocks {
    static constexpr int value = !SWEEP || sizeof(S) == 8 ? 2 : MODE == 1 ? 2 : 3;
};

// MODE: 1 = RK3 stage 3 (fluxes of buffer 2), 2 = RK3 final (buffer 3),
// 3 = RK1 update, 4 = EULER update, 5 = EULER_EQ update (buffer 2)
// PATH: FLUX_SWEEP or FLUX_GENERAL, the tiles of one kind per launch (a
// block given the other kind returns at once).
// TC: the default tile shape, compiled in; other shapes are read from the
// arguments and give every node the same bits (1024^2 Couette FP32, ms per
// step: 0.28 compiled in, 0.48 to 0.57 for other shapes).
// LAW: samples may have a viscosity law (macro_from_sums); only FP64 has
// instances without (a 1001 x 101 plate 3 % faster, FP32 RK1 1 % slower).
// NEXT: RK3's final phase goes on to the next step's stages (joins).
//
// What bounds it (64-sample ensemble, 3.5 M nodes; per-node sweeps with a
// barrier per four directions before): FP32 stage 3 535 us, waits on
// dependencies and loads at 16 warps per SM, issue slots 49 % used, FMA pipe
// 47 %, DRAM 33 % at the 413 of 416 bytes a node it has to move; the final
// phase with the next step's stages 380 us, issue slots 58 %, FMA pipe 56 %,
// DRAM 45 %.  FP64 789 and 433 us, FP64 pipe 62 and 61 %, DRAM 48 and 59 %.
// Steps of the same ensemble: FP32 1.98 -> 1.29 ms (5.1 M nodes), FP64 of 16
// samples 1.99 -> 0.99 ms (2.2 M nodes).
template <class S, int MODE, int PATH, bool TC, bool LAW, bool NEXT>
__global__ void __launch_bounds__(256, FluxBlocks<S, MODE, PATH == FLUX_SWEEP && TC>::value) k_flux(KArgs<S> a)
{
    using V = Pair<S>;
    extern __shared__ __align__(128) unsigned char smem_dyn[];
    __shared__ double red[32];
    __shared__ SampleParams s_sp;  // kept out of registers: read as needed
    __shared__ Tile s_tile;
    constexpr bool SWEEP = PATH == FLUX_SWEEP;
    const int TX = TC ? TILE_CX : a.tx, TY = TC ? TILE_CY : a.ty, NT = TX * TY;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    V *sm = reinterpret_cast<V *>(smem_dyn + ((128 - (smem_u32(smem_dyn) & 127)) & 127));
    const Tile t = a.tiles[blockIdx.x];
    if (tile_sweep(t) != SWEEP) return;
    constexpr int PH = MODE == 2 ? 2 : 1;
    const CUtensorMap *maps = a.tmaps + MAPS_PER_SAMPLE * t.sample + (PH == 1 ? 0 : 3);
    const S *stage = PH == 1 ? a.buf2 : a.buf3;
    const int PR = TX + 1, PP = part_pairs(TX, TY);
    constexpr FluxSmem LC = flux_smem<S>(TILE_CX, TILE_CY, true, true, 12);
    FluxSmem L = LC;
    if constexpr (!TC) L = flux_smem<S>(TX, TY, false, SWEEP, SWEEP ? a.slots : 0);
    uint64_t *bars = reinterpret_cast<uint64_t *>(sm + L.bar_off);
    S *save = reinterpret_cast<S *>(sm + L.wall_off);

    if constexpr (TC && SWEEP) {
        // each warp asks for its own boxes, and alone waits for them
        if (lane == 0) {
            const int ix = warp >= 4 ? warp + 1 : warp < 2 ? 1 + 2 * warp : 5 + 2 * warp;
            mbar_init(&bars[ix - 1], 1);
            if (warp < 4) mbar_init(&bars[ix], 1);
            fence_mbar_init();
            pdl_wait();
            issue_warp<S>(t, maps, sm, bars, warp);
        }
        // the warp's other lanes poll the barriers only once they are set up
        // (the block barrier below is not on every path)
        __syncwarp();
    } else if constexpr (SWEEP) {
        if (tid == 0) {
            for (int b = 0; b < a.slots; ++b) mbar_init(&bars[b], 1);
            fence_mbar_init();
        }
    }
    {
        const SampleParams *gsp = a.samples + t.sample;
        for (int k = tid; k < (int)(sizeof(SampleParams) / 4); k += NT)
            reinterpret_cast<int *>(&s_sp)[k] = reinterpret_cast<const int *>(gsp)[k];
        if (tid == 0) s_tile = t;
    }
    pdl_wait();
    // (what a plain tile's sweeps need is in the tile itself)
    if (!TC || !SWEEP || flux_early<S>(MODE) || (t.kind & TILE_FIX)) __syncthreads();
    const SampleParams &sp = s_sp;
    bool ok = true;
    if constexpr (TC && SWEEP) {
        // the rows of the state that the per-node half will read, into L2
        // (3 % of an FP64 step; FP32 gains nothing)
        if constexpr (sizeof(S) == 8) {
            const V *p = pair_base(a.state, sp) + (t.y0 + warp) * sp.pitch + t.x0 + lane;
            if ((lane & 7) == 0 && t.y0 + warp < sp.ny)
                for (int i = 0; i < NQ; ++i) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + i * (int)sp.plane));
        }
        ok = sweep_tile<S>(t, sp, stage, sm, save, bars, warp, lane);
    } else if constexpr (SWEEP) {
        const int fm = tile_fm(t.kind), gx = (t.kind & TILE_GHOST) ? GHOST_X : 0;
        for (int i0 = 1, r = 0; i0 <= 12; i0 += a.slots, ++r) {
            const int nd = min(a.slots, 13 - i0);
            if (tid == 0) {
                fence_proxy_async_smem();
                for (int d = 0; d < nd; ++d)
                    issue_box<S>(sm + d * L.slot_pairs, maps, t.x0, t.y0, gx, TX, TY, i0 + d, &bars[d]);
            }
            // every thread waits for every copy of the round
            for (int d = 0; d < nd; ++d) ok = mbar_wait_bounded(&bars[d], r & 1, TMA_WAIT_POLLS) && ok;
            if (t.kind & TILE_FIX) {
                for (int d = 0; d < nd; ++d) fix_box<S>(sm + d * L.slot_pairs, sp, stage, t, TX, TY, i0 + d, tid, NT);
                __syncthreads();
            }
            V *parts = sm + L.part_off;
            if (sizeof(S) == 8 ? fm != 0 : fm == 1)
                sweep_block<S, 1>(t, sp, sm, L.slot_pairs, parts, save, TX, TY, i0, nd, tid, NT);
            else if (fm == 2)
                sweep_block<S, sizeof(S) == 4 ? 2 : 1>(t, sp, sm, L.slot_pairs, parts, save, TX, TY, i0, nd, tid, NT);
            else sweep_block<S, 0>(t, sp, sm, L.slot_pairs, parts, save, TX, TY, i0, nd, tid, NT);
            __syncthreads();
        }
    }
    if (!ok) atomicOr(&a.status[a.tiles[blockIdx.x].sample], STATUS_TIMEOUT);
    const int tx = tid % TX, ty = tid / TX;
    const NodeParts<S, TC && SWEEP> part{TC && SWEEP ? sm : sm + L.part_off, ty * PR + tx, PP};
    if constexpr (!SWEEP) {
        const StageView<S> v{stage + sp.state_off, a.nflags + sp.node_off, (int)sp.plane, sp.pitch};
        face_parts<S>(t, sp, v, a.template alpha_as<S>() + sp.node_off, a.fref + NPL * t.sample, sm + L.part_off,
                      sm + L.wall_off, TX, TY, tid, NT);
    }
    node_phase<S, MODE, SWEEP, LAW, NEXT>(a, s_tile, sp, part, save, red, TX, NT, tid);
}

// ----------------------------------------------------------------- launchers
// calls f with the mode as a compile-time value
template <class F>
void with_mode(int mode, F f)
{
    switch (mode) {
    case 1: f(std::integral_constant<int, 1>()); break;
    case 2: f(std::integral_constant<int, 2>()); break;
    case 3: f(std::integral_constant<int, 3>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    default: f(std::integral_constant<int, 5>()); break;
    }
}

// calls f with every instance that launch_flux can take
template <class S, class F>
void with_kernel(int mode, bool sweep, bool def, bool constant_mu, bool next, F f)
{
    with_mode(mode, [&](auto m) {
        constexpr int M = decltype(m)::value;
        constexpr bool NX = M == 2 && joins<S>(TILE_CX, TILE_CY);
        constexpr bool L0 = sizeof(S) == 4;
        if (sweep && !def) f(k_flux<S, M, FLUX_SWEEP, false, true, false>);
        else if (!sweep) f(next ? k_flux<S, M, FLUX_GENERAL, false, true, NX> : k_flux<S, M, FLUX_GENERAL, false, true, false>);
        else if (next) f(constant_mu ? k_flux<S, M, FLUX_SWEEP, true, L0, NX> : k_flux<S, M, FLUX_SWEEP, true, true, NX>);
        else f(constant_mu ? k_flux<S, M, FLUX_SWEEP, true, L0, false> : k_flux<S, M, FLUX_SWEEP, true, true, false>);
    });
}

template <class S>
cudaError_t launch_flux(int mode, const KArgs<S> &a, int ntiles, int path, cudaStream_t st)
{
    KArgs<S> k = a;
    const bool def = k.tx == TILE_CX && k.ty == TILE_CY, sweep = path == FLUX_SWEEP;
    k.slots = def ? 12 : flux_slots<S>(k.tx, k.ty);
    const size_t sm = flux_smem_bytes_t<S>(k.tx, k.ty, sweep);
    cudaError_t e = cudaSuccess;
    with_kernel<S>(mode, sweep, def, k.constant_mu, k.next,
                   [&](auto *kernel) { e = launch_step_kernel(kernel, ntiles, k.tx * k.ty, sm, st, !k.phased, k); });
    return e;
}

template <class S>
cudaError_t prepare_flux()
{
    const int maxsm = 224 * 1024;
    cudaError_t e = cudaSuccess;
    for (int mode = 1; mode <= 5; ++mode)
        for (int k = 0; k < 16; ++k)
            with_kernel<S>(mode, k & 1, k & 2, k & 4, k & 8, [&](auto *kernel) {
                if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, maxsm);
            });
    return e;
}

}  // namespace uqlbm
