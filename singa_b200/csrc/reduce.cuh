// Internal interface of the column sums, used by the loss head.
#pragma once
#include "common.cuh"

namespace sgb {

// The column sums of M and, beside them, the sum of x's nrow elements: what
// sgb_sum_all_f32 and sgb_sum_rows_f32 give, bit for bit, by one launch where each
// of them is one (32x1000 with the head in front: 6.2 -> 5.3 us).  Doing the whole
// head in one CTA as well is slower from 64 rows on (64x10: 6.6 us, 256x10: 19.3,
// against 5.0 and 5.3): rows have to wait for one another there.
int sum_rows_beside_total(const float* M, float* v, size_t nrow, size_t ncol, const float* x, float* total, void* ws,
                          size_t ws_bytes, void* stream);

}  // namespace sgb
