// Whole-block entry points: workspace layout and device flag codes.
#pragma once

#include "common.cuh"

// Device flag word (first 16 bytes of every workspace): [0] code, [1..3] detail.
enum {
    LMOE_FLAG_BAD_EXPERT_ID = 0x1,
    LMOE_FLAG_WAIT_TIMEOUT = 0x2,
    LMOE_FLAG_BAD_INDEX = 0x4,
};
// What follows it when a prompt's routing went through the filter (route_filter.cu): [LMOE_CONTROL_LEFT] the experts that
// the bounds left, over all tokens of the call, [LMOE_CONTROL_DENSE] the tokens that got all their logits from route_dense_kernel.
enum { LMOE_CONTROL_LEFT = 4, LMOE_CONTROL_DENSE = 5, LMOE_CONTROL_WORDS = 8 };

// seam checks shared by the mat-vec and grouped-GEMM entry points (api.cu)
lmoe_status lmoe_id_shape_check(const lmoe_expert_stack *stack, const void *x, int64_t t, int64_t x_per_row,
                                int64_t k, const void *ids, int64_t t_ids, int64_t top_k, const void *out);

lmoe_status lmoe_combine_check(int64_t seq, int64_t top_k, int64_t n_out);

// Rows of one grouped product (mm_id.cu): `rows` routed rows over n_expert lists, `extra` rows of the shared expert behind
// them, row tiles of nt rows.
struct MmRows {
    int64_t rows, extra, max_tiles;
    int n_expert, nt;
};
