// row_blocks.h -- rows that start anywhere, read as the 16-byte blocks that
// cover them (piv_fp32.cuh): which rows' blocks leave the frame.
#pragma once
#include <cstddef>
#include <cstdint>

namespace opiv {

#ifdef __CUDACC__
#define OPIV_HD __host__ __device__
#else
#define OPIV_HD
#endif

// The blocks of a row of `row_bytes` (a multiple of 16) that starts at `row`:
// row_bytes / 16 of them from the block it starts in, and one more unless it
// starts on a block.  True if one of them has a byte outside the frame's
// [lo, lo + frame_bytes): up to 15 before the first pixel or after the last.
OPIV_HD inline bool blocks_leave(uintptr_t row, size_t row_bytes, uintptr_t lo, size_t frame_bytes)
{
    const uintptr_t mis = row & 15, first = row - mis;
    return mis != 0 && (first < lo || first + row_bytes + 16 > lo + frame_bytes);
}

// Bytes from a frame's first pixel to its last.
OPIV_HD inline size_t frame_extent(int img_w, int img_h, size_t pitch, size_t px)
{
    return (size_t)(img_h - 1) * pitch + (size_t)img_w * px;
}

// Whether a block of a row of a grid of w x w windows may leave the frame:
// of all windows, the first one's first row has the lowest address and the last
// one's last row the highest.
OPIV_HD inline bool grid_blocks_leave(uintptr_t lo, int img_w, int img_h, size_t pitch, size_t px, int w, int gx0, int gy0,
                                      int gdx, int gdy, int64_t nx, int64_t ny)
{
    const size_t extent = frame_extent(img_w, img_h, pitch, px), row_bytes = (size_t)w * px;
    const size_t y1 = (size_t)(gy0 + (ny - 1) * gdy + w - 1), x1 = (size_t)(gx0 + (nx - 1) * gdx);
    return blocks_leave(lo + (size_t)gy0 * pitch + (size_t)gx0 * px, row_bytes, lo, extent) ||
           blocks_leave(lo + y1 * pitch + x1 * px, row_bytes, lo, extent);
}

#undef OPIV_HD

}  // namespace opiv
