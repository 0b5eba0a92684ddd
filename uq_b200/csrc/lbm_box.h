// The halo boxes of the stencil kernels: their shapes, shared by the kernels
// (lbm_flux.cuh) and by the host, which encodes their TMA descriptors.
#pragma once

#include "lbm_device.cuh"
#include "lbm_kernels.h"

#include <cuda.h>
#include <cudaTypedefs.h>

namespace uqlbm {

constexpr int HALO = 3;

// Box columns.  FP32: a copy starts on a 16-byte boundary, so the halo is 4
// nodes on the left, and rows of tx + 10 pairs let the 8 rows of an x sweep
// read 16 bytes each without bank conflicts; FP64 (16-byte pairs): any start,
// and an odd row length does the same.
template <class S>
struct BoxCols {
    static constexpr int left = sizeof(S) == 4 ? 4 : 3;
    static constexpr int extra = sizeof(S) == 4 ? 10 : 7;  // 2^k + extra columns in all
};

// boxes by direction: x directions need the tile's rows, y directions its
// columns, diagonals both halos
enum BoxShape { BOX_X = 0, BOX_Y = 1, BOX_XY = 2 };
__host__ __device__ constexpr int box_shape(int i) { return lat_ey(i) == 0 ? BOX_X : lat_ex(i) == 0 ? BOX_Y : BOX_XY; }

template <class S>
__host__ __device__ constexpr int box_width(int shape, int tx)
{
    return shape == BOX_Y ? tx : tx + BoxCols<S>::extra;
}
__host__ __device__ constexpr int box_height(int shape, int ty) { return shape == BOX_X ? ty : ty + 2 * HALO; }
// FP64 boxes wider than a TMA box may be in 8-byte elements (256): the map
// gets the pair as a dimension of its own
template <class S>
__host__ __device__ constexpr bool box_map_4d(int tx)
{
    return sizeof(S) == 8 && 2 * box_width<S>(BOX_XY, tx) > 256;
}

// TMA descriptor of one buffer of a sample, its 13 planes as a 3D tensor
// (x, y, plane), for boxes of bw x bh nodes of one plane.  The elements are
// moved as 8-byte words: an FP32 pair, or one value of an FP64 pair (then x
// counts values; four: the pair as a dimension of its own).  With ghost
// columns the tensor starts at the left ghosts and spans the pitch (boxes at
// the x edges then read the images); else it is the domain, and boxes read
// zeros beyond it.
template <class S>
bool encode_map_t(PFN_cuTensorMapEncodeTiled_v12000 enc, const SampleParams &p, unsigned char *buf, int bw, int bh,
                  bool four, CUtensorMap *map)
{
    const cuuint64_t pair = 2 * sizeof(S), nx = (cuuint64_t)(p.gx ? p.pitch : p.nx);
    unsigned char *base = buf + (size_t)(p.state_off - 2 * p.gx) * sizeof(S);
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    if (four) {
        const cuuint64_t dims[4] = {2, nx, (cuuint64_t)p.ny, (cuuint64_t)NQ};
        const cuuint64_t strides[3] = {pair, p.pitch * pair, (cuuint64_t)p.plane * pair};
        const cuuint32_t box[4] = {2, (cuuint32_t)bw, (cuuint32_t)bh, 1};
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    }
    const cuuint32_t w = (cuuint32_t)(pair / 8);
    const cuuint64_t dims[3] = {nx * w, (cuuint64_t)p.ny, (cuuint64_t)NQ};
    const cuuint64_t strides[2] = {p.pitch * pair, (cuuint64_t)p.plane * pair};
    const cuuint32_t box[3] = {(cuuint32_t)bw * w, (cuuint32_t)bh, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The MAPS_PER_SAMPLE descriptors of a sample.
template <class S>
bool encode_box_maps_t(PFN_cuTensorMapEncodeTiled_v12000 enc, const SampleParams &p, unsigned char *buf2,
                       unsigned char *buf3, int tx, int ty, CUtensorMap *maps)
{
    for (int b = 0; b < 6; ++b)
        if (!encode_map_t<S>(enc, p, b < 3 ? buf2 : buf3, box_width<S>(b % 3, tx), box_height(b % 3, ty),
                             box_map_4d<S>(tx), &maps[b]))
            return false;
    return true;
}

inline bool encode_box_maps(PFN_cuTensorMapEncodeTiled_v12000 enc, bool f64, const SampleParams &p, unsigned char *buf2,
                            unsigned char *buf3, int tx, int ty, CUtensorMap *maps)
{
    return f64 ? encode_box_maps_t<double>(enc, p, buf2, buf3, tx, ty, maps)
               : encode_box_maps_t<float>(enc, p, buf2, buf3, tx, ty, maps);
}

}  // namespace uqlbm
