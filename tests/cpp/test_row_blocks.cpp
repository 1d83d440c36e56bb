// Every row of every window of small frames at every base address and several
// pitches: where blocks_leave says that a row's blocks stay, all the bytes that
// the block loads read lie in the frame; where it says that one leaves, one does.
#include <cstdio>
#include <initializer_list>

#include "row_blocks.h"

int main()
{
    long rows = 0, leaving = 0;
    for (size_t px : { 1, 2, 4 })
        for (int ia : { 16, 32 })
            for (int img_w : { ia, ia + 1, ia + 5, ia + 16, 3 * ia })
                for (int img_h : { ia, ia + 3 })
                    for (size_t pad : { 0, 1, 3, 16 })
                        for (uintptr_t base = 4096; base < 4096 + 16; base += px) {
                            const size_t pitch = ((size_t)img_w + pad) * px, bytes = (size_t)ia * px;
                            const uintptr_t end = base + opiv::frame_extent(img_w, img_h, pitch, px);
                            // the grid rule against its windows' rows
                            for (int step : { 1, 5, 16 }) {
                                const int nx = (img_w - ia) / step + 1, ny = (img_h - ia) / step + 1;
                                const int gx0 = (img_w - ia - step * (nx - 1)) / 2, gy0 = (img_h - ia - step * (ny - 1)) / 2;
                                bool any = false;
                                for (int j = 0; j < ny; ++j)
                                    for (int i = 0; i < nx; ++i)
                                        for (int y : { 0, ia - 1 })
                                            any = any || opiv::blocks_leave(
                                                base + (gy0 + j * step + y) * pitch + (gx0 + i * step) * px, bytes, base, end - base);
                                if (any != opiv::grid_blocks_leave(base, img_w, img_h, pitch, px, ia, gx0, gy0, step, step, nx, ny)) {
                                    std::printf("grid: px %zu ia %d %dx%d pad %zu base %zu step %d\n", px, ia, img_w, img_h, pad,
                                                (size_t)base, step);
                                    return 1;
                                }
                            }
                            if (end != base + (img_h - 1) * pitch + img_w * px) return 1;
                            for (int y = 0; y < img_h; ++y)
                                for (int x = 0; x + ia <= img_w; ++x) {
                                    const uintptr_t row = base + y * pitch + x * px, block = row & ~(uintptr_t)15;
                                    const size_t n = bytes / 16 + (row != block);
                                    const bool out = block < base || block + 16 * n > end;
                                    const bool said = opiv::blocks_leave(row, bytes, base, end - base);
                                    // an aligned row's blocks are the row itself
                                    if (said != out) {
                                        std::printf("px %zu ia %d %dx%d pad %zu base %zu y %d x %d: %d %d\n", px, ia, img_w,
                                                    img_h, pad, (size_t)base, y, x, said, out);
                                        return 1;
                                    }
                                    ++rows;
                                    leaving += said;
                                }
                        }
    if (leaving == 0) return 1;
    std::printf("ok %ld rows, %ld leave\n", rows, leaving);
    return 0;
}
