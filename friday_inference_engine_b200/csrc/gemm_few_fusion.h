// Optional work at the two ends of the 32-bit product of few rows (gemm_simt_few); a zeroed struct asks for none.  In a one-token
// step of a small model every kernel costs its launch and little else, and the neighbours that go into the products are
// half of them.
#pragma once

struct GemmFewFusion {
    // (1) RMSNorm of the input rows: the product of x / sqrt(mean x^2 + eps) * norm_w (null: of x as it is).
    const void* norm_w;
    int norm_w_dtype;
    float eps;
    // (2) A gated unit: columns 2 f and 2 f + 1 of the product are gate and up of result column f (0: none; as fr_gated).
    int act;
    float act_limit, act_slope;
    // (3) Rotary encoding and cache write: the result is [q heads | k heads | v heads] of hd columns each (nq 0: none).  Row r belongs
    // to sequence row_seq[r] (negative: left as it is) at position row_pos[r]; with denom (rot / 2 denominators) the pairs
    // (i, i + rot / 2) of every q and k head are rotated by pos / denom[i]; with pools, k and v also go to the cache row that
    // `table` gives the position.
    const int* row_seq;
    const int* row_pos;
    const float* denom;
    float* k_pool;
    float* v_pool;
    const int* table;
    int rot, nq, nkv, hd, table_width, page;
    // (4) Not zero: no kernel writes the weights any more; they may be read while the kernel before this one still runs.
    int fixed_weights;
};
