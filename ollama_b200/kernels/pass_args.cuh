// Arguments of the products of unit-ordered matrices in 16-bit rows.
#pragma once
#include "common.cuh"

// Products of unit-ordered matrices (gemm_sk.cu).
struct SgSeg {
    const uint8_t* w;     // units [n / 16][k / 256][unit bytes]
    const float* bias;    // [n] or null
    int type;             // WT_Q4_K or WT_Q6_K
    int n;                // rows, a multiple of 16
    int out_off;          // column of row 0 in the output row
    int tile0;            // first 16-row tile of this matrix in the launch (filled in by the launcher)
};

struct SgArgs {
    SgSeg seg[4];
    int nseg, k, nb;
    const uint8_t* x;     // chunks of b2_rows16
    int mode;             // 0: out = y, 1: out += y, 2: out[b][i] = act(y[2i], y[2i+1])
    float* out;
    int ldo, act;
    float alpha, limit;
    float* ws;            // [groups of b2_gemv_sk_max_groups][512]
    unsigned* flags;
    int* status;
    int tiles, ring, slot_bytes, x_slots;      // filled in by the launcher
};

struct Rows16Args {
    const void* x;        // [nb][ldx]
    int ldx;              // elements
    int bf16;             // 0: fp32 rows, 1: bf16 rows
    const float* norm_w;  // RMSNorm weight or null
    float eps;
    int k;
    uint8_t* out;         // [k / 256][ceil(nb / 8)][SG_CHUNK] regrouped: per 256-block all values, then all sums, then all scales
};
