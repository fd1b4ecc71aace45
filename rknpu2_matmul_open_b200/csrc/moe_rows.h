// moe_rows.h -- how the input rows of one routed-experts run reach the device: pulled by the intake kernel out of the
// workspace's page-locked piece, or copied by the driver; and how many rows the kept launches cover.  Host arithmetic only.
#pragma once
#include <stddef.h>

namespace rkb200 {

// Rows up to this size are staged in page-locked memory and read from there by the intake kernel; larger ones are copied
// from the caller's array by the driver (one token: the copy engine would cost another call and its own start, 4 + 2 us of
// about 30; 512 KB: 40 us against 44; 2 MB: 148 against 136).
constexpr size_t MOE_PULL_MOST = size_t(512) << 10;

// Bytes of input rows the page-locked piece of a workspace has room for (fp32 rows are the larger kind).
inline size_t moe_piece_row_bytes(int max_rows, int H)
{
    const size_t row = size_t(H) * 4, all = size_t(max_rows) * row, most = MOE_PULL_MOST > row ? MOE_PULL_MOST : row;
    return all < most ? all : most;
}

struct MoeRowPlan {
    bool pull;        // the rows are staged in the page-locked piece
    int level;        // kind of the launches: the grid's rows depend on it, on the kind of rows and on `pull` alone
    int grid_rows;    // rows the launches cover, at least the run's
};
// The grid is rounded up to a power of two so that few kept launches serve every row count.  The intake kernel requests an
// fp32 row of its grid before it knows whether the run has that row, so a grid that reads from the page-locked piece ends
// with the rows the piece can hold.  (The device copy of the rows has room for max_rows.)
inline MoeRowPlan moe_row_plan(int rows, int max_rows, int H, bool f32)
{
    MoeRowPlan p{size_t(rows) * H * (f32 ? 4 : 1) <= MOE_PULL_MOST, 0, 0};
    while ((1 << p.level) < rows) ++p.level;
    p.grid_rows = (1 << p.level) < max_rows ? 1 << p.level : max_rows;
    if (p.pull && f32) {
        const int held = int(moe_piece_row_bytes(max_rows, H) / (size_t(H) * 4));
        if (p.grid_rows > held) p.grid_rows = held;
    }
    return p;
}

} // namespace rkb200
