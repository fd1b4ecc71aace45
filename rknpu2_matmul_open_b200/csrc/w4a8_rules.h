// w4a8_rules.h -- rules of the W4A8 dispatch that are plain arithmetic on sizes.  Host only, no CUDA.
#pragma once
#include <stddef.h>

#include "persist_plan.h"

namespace rkb200 {

// Whether a blocking call's kernel stores its [M][cols] result of `elem` bytes each straight into page-locked host memory
// instead of leaving it to the copy engine.  `family`: the kernel family that runs the call (5 decode, 3 split-K, others in
// two launches).
//   * The decode kernel writes every element once, 32 neighbouring ones per warp: rows that do not start on a sector cost it
//     nothing visible (4 x 4911 fp32 26 us against 33 copied, 4 x 14330 32 against 38, 8 x 4911 at K = 11008 47 against 55).
//   * The split-K kernel stores four neighbours at once where the row length allows it (8 x 2900 binary16 26 us against 32
//     copied); element by element the bus takes them slowly (8 x 4911 58 us against 33), so then small results only.
//   * The single-kernel families up to 1 MB (8 x 28672 fp32 44 us against 49, into an ordinary array 84 against 100).  The
//     others write pieces of 64 bytes, which the bus takes more slowly: from 128 KB on the copy engine is as fast, and rows
//     that do not start on a sector leave it in pieces of sectors (13 x 4910 binary16 64 us against 38, 13 x 4912 34).
constexpr size_t RESULT_OVER_BUS_MOST = size_t(1) << 20;
inline bool result_over_bus(int family, int M, size_t cols, size_t elem)
{
    const size_t bytes = size_t(M) * cols * elem;
    const bool single = family == 5 || family == 3;
    if (bytes > (single ? RESULT_OVER_BUS_MOST : size_t(128) << 10)) return false;
    if (M == 1 || family == 5 || cols * elem % 32 == 0 || (family == 3 && cols % 4 == 0)) return true;
    return bytes <= (elem == 2 ? size_t(40) << 10 : size_t(64) << 10);
}

// 9..16 tokens of small weights: whether one launch (the split-K kernel, whose every cluster scans all of the rows) is left for
// two (quantise, ring).  For binary16 rows that allow 16-byte loads one launch is the faster at every count (16 tokens, 4096 ->
// 4096 10.2 us against 11.0, 4096 -> 1024 8.4 against 9.5, 1024 -> 14336 9.6 against 9.9; at worst 5504 -> 2112 10.7 against
// 10.2).  fp32 rows are twice the scan: 13 tokens and more take two (13 tokens 2048 -> 2048 9.3 against 8.7, 4096 -> 4096 11.7
// against 10.4, 16 tokens 2048 -> 8192 12.3 against 9.7; 12 tokens 8.8 against 8.7, 4096 -> 1024 8.4 against 9.3).  Rows that
// are loaded element by element sooner still: binary16 from 11 tokens (10 tokens 1500 -> 2048 7.9 against 9.5, 2044 -> 4096
// 11.6 against 11.0; 12 tokens 3070 -> 4911 13.1 against 11.5, 16 tokens 15.9 against 11.7), fp32 from 9 (3070 -> 4911 16.6
// against 12.1, 1025 -> 1024 11.5 against 9.6).
inline bool mid_batch_takes_ring(int M, int K, bool half)
{
    const bool wide = K % 8 == 0;
    return half ? !wide && M > 10 : M > (wide ? 12 : 8);
}

} // namespace rkb200
