// One prompt pass through a run of dense layers, launched from native code.
//
// A layer is eight launches (norm, q/k/v, rotation + cache append, attention, output, norm, gate/up, down) of 5 to 100 us at short and middling lengths; made one by one
// from Python they cost about 12 us each, so that 7 drafted tokens of 12 layers took 1.96 ms for 1.1 ms of kernels.  From here a launch costs what the driver takes.
// The caller's buffers are the layers' own: nothing is allocated or kept.
#include "pass_args.cuh"

extern "C" {
int b2_rmsnorm_bf16(const NormCastArgs* a, int rows, int pdl, cudaStream_t st);
int b2_rope_kv(const RopeKvArgs* a, int nt, int pdl, cudaStream_t st);
int b2_attn_prefill_tc(const AttnPrefillArgs* a, int head_dim, int n_slots, int pdl, cudaStream_t st);
int b2_attn_prefill_q8(const AttnPrefillArgs* in, int head_dim, int n_slots, void* scratch, long long halves, int pdl, cudaStream_t st);
int b2_attn_prefill(const AttnPrefillArgs* a, int head_dim, cudaStream_t st);
int b2_gemm_bf16(const void* a, const void* b, int m, int n, int k, float* out, int ldo, const float* bias, int accumulate, int pdl, float* ws,
                 long long ws_floats, cudaStream_t st);
int b2_gemm_bf16_glu(const void* a, const void* b, int m, int n, int k, void* out, int ldo, const float* bias, int act, float alpha, float limit, int pdl, cudaStream_t st);
int b2_rows16(const Rows16Args* in, int nb, int pdl, cudaStream_t st);
int b2_gemm_sk(const SgArgs* in, int max_ctas, int pdl, cudaStream_t st);
}

struct PassLayer {
    const float *attn_norm, *ffn_norm;
    const void *wqkv, *wo, *gu, *down;            // resident 16-bit matrices, or null with units
    const float *bqkv, *bo, *bgu, *bdown;
    SgSeg units[6];                               // q, k, v, output, gate/up, down in unit order, where the pass may use them
    const float *q_norm, *k_norm, *sinks, *inv_freq;
    float mscale;
    int window;
    __half *k_cache, *v_cache, *k_scale, *v_scale;
};

struct PassSeg {
    int row0, rows, slot, pos0;                   // rows of one sequence, from position pos0 on
};

struct PassArgs {
    int rows, d, n_heads, n_kv_heads, hd, n_rot, neox, n_ctx, n_slots, ff, causal, act;
    float eps, scale, softcap, alpha, limit;
    const int *positions, *slots;                 // [rows], device
    float *x, *qkv, *q;                           // residual stream [rows][d]; [rows][(H + 2 Hkv) hd]; [rows][H hd]
    void *o, *h;                                  // bf16 [rows][H hd], [rows][d]
    void* f;                                      // bf16 [rows][ff], units: fp32
    uint8_t* x16;                                 // units: b2_rows16_bytes(min(rows, 64), widest row)
    float* ws;                                    // units: workspace of b2_gemm_sk, otherwise scratch of b2_gemm_bf16
    long long ws_floats;
    int* status;
    int units, tc, pdl;                           // tc: attention on tcgen05 where it applies
    void* kv16;                                   // int8 caches: scratch of b2_attn_prefill_q8, or null
    long long kv16_halves;
    int launches;                                 // out
};

namespace {

constexpr int UNIT_ROWS = 64;

// Rows of `x` (fp32, or bf16 when ldx counts those), normalised with `w` where given, times unit-ordered matrices.
int unit_product(const PassArgs& a, const SgSeg* w, int n, const void* x, int bf16, int k, const float* norm, float* out, int ldo, int mode, int& count, cudaStream_t st) {
    for (int r = 0; r < a.rows; r += UNIT_ROWS) {
        const int nb = a.rows - r < UNIT_ROWS ? a.rows - r : UNIT_ROWS;
        const Rows16Args ra{(const uint8_t*)x + (size_t)r * k * (bf16 ? 2 : 4), k, bf16, norm, a.eps, k, a.x16};
        int rc = b2_rows16(&ra, nb, a.pdl, st);
        if (rc) return rc;
        SgArgs s = {};
        int off = 0;
        for (int i = 0; i < n; i++) {
            s.seg[i] = w[i];
            s.seg[i].out_off = off;
            off += w[i].n;
        }
        s.nseg = n;
        s.k = k;
        s.nb = nb;
        s.x = a.x16;
        s.mode = mode;
        s.out = out + (size_t)r * ldo;
        s.ldo = ldo;
        s.act = a.act;
        s.alpha = a.alpha;
        s.limit = a.limit;
        s.ws = a.ws;
        s.status = a.status;
        rc = b2_gemm_sk(&s, 0, a.pdl, st);
        if (rc) return rc;
        count += 2;
    }
    return 0;
}

}  // namespace

// Enqueues layers 0 .. n - 1 on `st`; `segs`: host array.  Returns a cudaError_t value.
B2_API int b2_prefill_pass(const PassLayer* layers, int n, PassArgs* io, const PassSeg* segs, int n_segs, cudaStream_t st) {
    const PassArgs& a = *io;
    if (n < 1 || a.rows < 1 || n_segs < 1) return (int)cudaErrorInvalidValue;
    const int qd = a.n_heads * a.hd, nq = (a.n_heads + 2 * a.n_kv_heads) * a.hd, late = a.pdl ? 2 : 0;
    int rc = 0, count = 0;
    for (int i = 0; i < n && !rc; i++) {
        const PassLayer& L = layers[i];
        const NormCastArgs n1{a.x, L.attn_norm, a.eps, a.d, 1, (__nv_bfloat16*)a.h}, n2{a.x, L.ffn_norm, a.eps, a.d, 1, (__nv_bfloat16*)a.h};
        if (a.units) {
            if ((rc = unit_product(a, L.units, 3, a.x, 0, a.d, L.attn_norm, a.qkv, nq, 0, count, st))) break;
        } else {
            if ((rc = b2_rmsnorm_bf16(&n1, a.rows, a.pdl, st))) break;
            if ((rc = b2_gemm_bf16(a.h, L.wqkv, a.rows, nq, a.d, a.qkv, nq, L.bqkv, 0, late, a.ws, a.ws_floats, st))) break;
        }
        const RopeKvArgs rope{a.qkv, a.positions, a.slots, L.inv_freq, L.q_norm, L.k_norm, a.eps, L.mscale, a.n_heads, a.n_kv_heads, a.hd, a.n_rot, a.neox, a.n_ctx, a.q,
                              L.k_cache, L.v_cache, L.k_scale, L.v_scale};
        if ((rc = b2_rope_kv(&rope, a.rows, a.pdl, st))) break;
        for (int s = 0; s < n_segs && !rc; s++) {
            const PassSeg& g = segs[s];
            const AttnPrefillArgs at{a.q + (size_t)g.row0 * qd, L.k_cache, L.v_cache, (__nv_bfloat16*)a.o + (size_t)g.row0 * qd, L.sinks, g.rows, a.n_heads, a.n_kv_heads, a.n_ctx,
                                     g.slot, g.pos0, g.pos0 + g.rows, a.causal, L.window, a.scale, a.softcap, L.k_scale, L.v_scale};
            rc = (int)cudaErrorNotSupported;
            if (a.tc && (a.hd == 64 || a.hd == 128))
                rc = !L.k_scale ? b2_attn_prefill_tc(&at, a.hd, a.n_slots, a.pdl, st)
                     : a.kv16   ? b2_attn_prefill_q8(&at, a.hd, a.n_slots, a.kv16, a.kv16_halves, a.pdl, st)
                                : (int)cudaErrorNotSupported;
            if (!rc && L.k_scale) count++;
            if (rc == (int)cudaErrorNotSupported) rc = b2_attn_prefill(&at, a.hd, st);      // nothing was launched
        }
        if (rc) break;
        if (a.units) {
            if ((rc = unit_product(a, L.units + 3, 1, a.o, 1, qd, nullptr, a.x, a.d, 1, count, st))) break;
            if ((rc = unit_product(a, L.units + 4, 1, a.x, 0, a.d, L.ffn_norm, (float*)a.f, a.ff, 2, count, st))) break;
            if ((rc = unit_product(a, L.units + 5, 1, a.f, 0, a.ff, nullptr, a.x, a.d, 1, count, st))) break;
            count += 1 + n_segs;
        } else {
            if ((rc = b2_gemm_bf16(a.o, L.wo, a.rows, a.d, qd, a.x, a.d, L.bo, 1, late, a.ws, a.ws_floats, st))) break;
            if ((rc = b2_rmsnorm_bf16(&n2, a.rows, a.pdl, st))) break;
            if ((rc = b2_gemm_bf16_glu(a.h, L.gu, a.rows, 2 * a.ff, a.d, a.f, a.ff, L.bgu, a.act, a.alpha, a.limit, late, st))) break;
            if ((rc = b2_gemm_bf16(a.f, L.down, a.rows, a.d, a.ff, a.x, a.d, L.bdown, 1, late, a.ws, a.ws_floats, st))) break;
            count += 7 + n_segs;
        }
    }
    io->launches = count;
    return rc;
}
