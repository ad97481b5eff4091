// Grid index construction (device).
#pragma once
#include "rknn_common.cuh"
#include <cstring>

namespace rknn {

// Bounding box of points as integer keys with the coordinates' order: x0, y0
// (least), x1, y1 (largest).
struct PointBox {
    unsigned key[4] = {0xffffffffu, 0xffffffffu, 0u, 0u};
};
inline float key_float(unsigned k)
{
    const unsigned u = (k & 0x80000000u) ? k & 0x7fffffffu : ~k;
    float f;
    memcpy(&f, &u, sizeof(f));
    return f;
}

// Folds n device points into *box and sets *bad when a coordinate is not
// finite (both on the device).
cudaError_t points_box(const float2* xy, int n, PointBox* box, int* bad, cudaStream_t st);

Grid make_grid(double x0, double y0, double x1, double y1, long long n, double per_cell, int max_side);

size_t grid_sort_bytes(int n, const Grid& g);
cudaError_t grid_sort(const float2* d_xy, const int* d_ids, int n, const Grid& g, char* ws,
                      float2* xy_s, int* ids_s, int* pos_of, int* start, cudaStream_t st);

// Boxes of the cells' points, and (*filled, on the device) how many cells have any.
cudaError_t cell_mbrs(const float2* xy_s, const int* start, const Grid& g, float4* mbr, int* filled, cudaStream_t st);

}  // namespace rknn
