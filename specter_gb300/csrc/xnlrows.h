// Rows a block of the FP32 nonlinear x pass (fast_launch.cuh, xnl).
#pragma once

namespace sg {

// rb: the largest number within the tile cap and the shared memory; pipelined: the length has a form that overlaps
// loads with transforms at 8 rows; pair: two blocks of 16 rows fit an SM.  16 rows with one block on an SM are
// slower than that form with two blocks of 8 (nx = 512, 512^2 x 513, four components: 8.2 against 6.1 ms); where
// two blocks of 16 fit (nx = 256) they are faster.  Only 512 is such a length.  A cap that was asked for is kept.
inline int xnl_rows(int rb, bool pipelined, bool pair, bool asked) {
    return pipelined && rb == 16 && !pair && !asked ? 8 : rb;
}

}  // namespace sg
