// Arguments of kernels that more than one source file launches.
#pragma once
#include "common.cuh"

struct RopeKvArgs {
    const float* qkv;        // [nt][(H + 2 Hkv) * hd]  (q | k | v)
    const int* positions;    // [nt]
    const int* slots;        // [nt]
    const float* inv_freq;   // [n_rot/2]
    const float* q_norm;     // [hd] or null
    const float* k_norm;     // [hd] or null
    float eps, mscale;
    int n_heads, n_kv_heads, hd, n_rot, neox, n_ctx;
    float* q_out;            // [nt][H][hd]
    __half* k_cache;         // [slots][Hkv][n_ctx][hd]  (int8 when the scale arrays are given)
    __half* v_cache;
    __half* k_scale;         // q8_0 cache: [slots][Hkv][n_ctx][hd/32] one f16 scale per 32 dims, or null for an f16 cache
    __half* v_scale;
};

struct NormCastArgs {
    const float* x;
    const float* w;
    float eps;
    int k, do_norm;
    __nv_bfloat16* out;
};

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
    float* ws;            // b2_gemm_sk_ws() floats, all bytes 255
    int* status;          // KStatus, written when a bounded wait gives up (may be pinned host memory)
    int tiles, ring, slot_bytes, x_slots;      // filled in by the launcher
};

struct Rows16Args {
    const void* x;        // [nb][ldx]
    int ldx;              // elements
    int bf16;             // 0: fp32 rows, 1: bf16 rows
    const float* norm_w;  // RMSNorm weight or null
    float eps;
    int k;
    uint8_t* out;         // [k / 256][ceil(nb / 16)][SG_CHUNK] regrouped: per 256-block all values, then all sums, then all scales
};

struct AttnPrefillArgs {
    const float* q;          // [T][H][D] fp32, rotary embedding already applied
    const __half* k_cache;   // [slots][Hkv][n_ctx][D]
    const __half* v_cache;
    __nv_bfloat16* out;      // [T][H * D]
    const float* sinks;      // [H] or null
    int T, H, Hkv, n_ctx;
    int slot, pos0;
    int kv_len;              // keys visible to the chunk: positions [0, kv_len)
    int causal;
    int window;              // 0 = none; key k is visible to query p when p - k < window
    float scale, softcap;
    const __half* k_scale;   // q8_0 cache (k_cache / v_cache hold int8): [slots][Hkv][n_ctx][D/32] scales, or null for f16
    const __half* v_scale;
};
