// Tensor maps for TMA, made on the host and kept per host thread (internal header).
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace tmw {

// Map over a row-major [rows, cols] matrix of 16-bit values with leading dimension ld (elements): boxes of
// box_rows x box_cols.  false: failed, with the error text set.
bool make_map_2d(CUtensorMap* map, const void* base, int dtype, int rows, int cols, int64_t ld, int box_rows, int box_cols,
                 CUtensorMapSwizzle swizzle);

// Strides (in elements) that the map of a [batch, heads, rows, dh] tensor uses.  The stride of an extent-1 axis is
// never used for addressing; it gets a harmless valid value.
struct MapStrides {
    int64_t row, head, batch;
    bool heads_first;  // the head axis has the smaller stride and comes before the row axis in the map
    bool ok;           // what a tensor map accepts: positive multiples of 16 bytes below 2^40 bytes
};
MapStrides map_strides(int batch, int heads, int rows, int dh, const int64_t stride[3]);

// Map over rows [0, rows) of a [batch, heads, *, dh] tensor of 16-bit values laid out by `m`: a box of box_rows rows x 64
// columns of one (batch, head), 128-byte swizzle.  Rows of a box at or beyond `rows` are filled with zeros on load and
// dropped on store.
bool make_map_4d(CUtensorMap* map, const void* base, int dtype, int batch, int heads, int rows, int dh, const MapStrides& m,
                 int box_rows);

}  // namespace tmw
