// Product of 1..64 rows with unit-ordered Q4_K / Q6_K matrices (the layout of gemv_sk.cu) in 16-bit activations, sm_100a.
//
// Decode steps of several sequences and short passes (drafted tokens, ends of prompts) multiply a few rows with matrices that stream from HBM once.
// The bound is that stream, so nothing else may cost more than it:
//   * Matrix instructions.  tcgen05.mma kind::f16, M = 128 matrix rows, N = the activation rows (16, 32, 48 or 64), K = a 256-block: its cost hardly depends on the rows (25 cycles
//     for 16 columns of K at 16 and 32 rows, 35 at 64), so the expansion of the codes is what an item costs beside its bytes.
//   * Weights.  An item is 128 matrix rows x 256 columns: eight units, which bulk copies bring into a ring that is filled before the grid-dependency wait.  16 warps expand them, one
//     unit of every second item each.  Codes become f16 in registers: a 4-bit code under the exponent of 1024 or 64 and one fused multiply-add give code x 6-bit scale exactly
//     (at most 945); of Q6_K code x scale is rounded once to 11 bits.  They go to tensor memory as the A operand (tcgen05.st.16x128b: lane (g, t) writes rows g and g + 8, words
//     t of every four, which is how the units are dealt to lanes), not to shared memory: 64 KB an item written there and read again would take longer than the item's 19 KB
//     from HBM.  K is permuted inside a 64-column group by that; the activations are stored in the same order.
//   * Activations.  b2_rows16 turns fp32 or bf16 rows (optionally RMS-normalised) into f16 values with one power-of-two scale per row and 256-block, in the 128-byte-swizzled
//     order of the B operand, so that a 256-block of all rows is one bulk copy.
//   * Sums.  The accumulators of a 256-block are read back by four warps (a thread a matrix row), which apply the block's d and the rows' scales in fp32 and add up; the Q4_K
//     minima are one more product per block (A: the minima twice, B: the rows' sums of 32 in two f16 parts) into columns of its own.
//     So neither operand is rounded to fewer bits than the f16 activation keeps (2^-12 of a block's largest value at worst, against 2^-8 of the int8 form and
//     2^-9 of products on bf16 copies): relative error of a product against 64 bits 2.1e-4 (Q4_K) and 2.6e-4 (Q6_K), int8 form 7e-3.
//   * Measured (Llama-8B layer, q/k/v + output + gate/up + down with the four b2_rows16 before them, Q4_K_M): 56 us at 2 rows, 57 at 16, 65 at 32, 87 at 64, where mma.sync fragments
//     expanded in registers took 74, 81, 113 and 226 (two launches), and 124 MB stream in 19.  What is left: 1100 cycles an item of 128 x 256 (expansion issues for 70 % of them), 2000
//     to 4000 cycles a launch until the first sums, and 3000 to exchange those of split groups.
//   * Work.  The launch's items are dealt out in equal contiguous shares, one CTA per SM.  The CTAs of a split group each finish a share of its values, adding the others' parts in a
//     fixed order.  Parts are handed over through a workspace without flags or fences (handed.cuh; bounded wait).  With the first CTA collecting everything behind flags, and all
//     warps watching flags that shared a line, a layer took 61, 64, 76 and 104 us.
#include "handed.cuh"
#include "pass_args.cuh"
#include "rows16.cuh"
#include "tc_common.cuh"

namespace {

using namespace tc;
constexpr int SG_TILES = 8;                                    // 16-row tiles of a group
// Warps: 16 that expand, in two teams of eight (a team takes every second item, a warp of it one group of 16 rows), 4 that add up, one each for the products of even and of
// odd items, the activations, the units of even and of odd items, and 3 that finish the rows of a group while the next one is under way.  72 registers a thread at the launch; the
// last eight warps leave 32 of theirs to those that add up.
constexpr int SG_EXPAND = 16, SG_SUM = 4, SG_FINISH = 3, SG_THREADS = (SG_EXPAND + SG_SUM + 5 + SG_FINISH) * 32;
enum { SG_MMA = SG_EXPAND + SG_SUM, SG_LOAD_X = SG_MMA + 2, SG_LOAD_W = SG_LOAD_X + 1, SG_LAST = SG_LOAD_W + 2 };
constexpr int SG_UNIT_Q4K = 2368, SG_UNIT_Q6K = 3360;
constexpr int SG_MAX_NT = SG_MAX_ROWS / 16;
constexpr int SG_WS_FLOATS = 128 * SG_MAX_ROWS;                // a CTA's share of the workspace
constexpr int SG_CTAS = 148;
constexpr int SG_MAX_SMEM = 224 * 1024;
constexpr int SG_SCALE_SLOTS = 8, SG_D_SLOTS = 8, SG_W_SLOTS = 10, SG_X_SLOTS = 4;
constexpr int SG_A_COLS = 136;                                 // TMEM columns of an item's expanded weights: 256 / 2 of codes x scales, 16 / 2 of minima
constexpr unsigned long long SG_WAIT_NS = 1000000000ull;

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait of about a second, as mbar_wait: a rolled loop, because the code of all roles has to stay in the instruction caches (unrolled waits, activations and halves of a
// block made it 136 KB).
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
#pragma unroll 1
    for (int i = 0; i < (1 << 22); i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (i > 128) __nanosleep(100);
    }
    return false;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t policy) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy) : "memory");
}
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t h2_add(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// two fp32 values as one operand of the packed instructions
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f2 pack2u(uint32_t a, uint32_t b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// f16 operands, both K-major
__host__ __device__ constexpr uint32_t sg_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24); }

// K-major operand without swizzle: cells of eight rows x 16 bytes are contiguous, `lbo` bytes apart along K and 128 along the rows.
__device__ __forceinline__ uint64_t desc_cells(uint32_t addr, uint32_t lbo) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(128 >> 4) << 32 | (uint64_t)1 << 46;
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {      // A in tensor memory
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ bool elect() {      // the same lane of a warp every time
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}
// 16 rows x 32 words: register 2 j of lane (g, t) is word 4 j + t of row g, register 2 j + 1 of row g + 8
__device__ __forceinline__ void tmem_st_16x128_x8(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]),
                 "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_16x128_x2(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x2.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
                   "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(taddr));
}

// f16x2 constants: 1024 or 64 under a code, and what takes it (times a scale) away again
constexpr uint32_t H_1024 = 0x64006400u, H_M1024 = 0xE400E400u, H_64 = 0x54005400u, H_M1024_M64 = 0xD400E400u, H_M1152 = 0xE480E480u, H_QUARTER = 0x34003400u, H_M288 = 0xDC80DC80u;

__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {      // (a & b) | c; written as such it became two instructions
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// one half twice: an operand form of the packed instructions
__device__ __forceinline__ uint32_t lower2(uint32_t v) {
    uint32_t d;
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tmov.b32 %0, {l, l};\n\t}" : "=r"(d) : "r"(v));
    return d;
}
__device__ __forceinline__ uint32_t upper2(uint32_t v) {
    uint32_t d;
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tmov.b32 %0, {h, h};\n\t}" : "=r"(d) : "r"(v));
    return d;
}

// 64 columns of a Q4_K unit (sub-blocks 2p from the low, 2p + 1 from the high nibbles) as 16 words: [j][row g, row g + 8]; `B`: byte of the first sub-block's scale in scg / sch.
// A low nibble stands under the exponent of 1024 (code + 1024), a high one under that of 64 (code + 64): both times the scale, less 1024 or 64 scales.
template <int B>
__device__ __forceinline__ void expand_q4k(const uint4 w, uint32_t scg, uint32_t sch, uint32_t (&r)[16]) {
    const uint4 v = make_uint4(w.x >> 8, w.y >> 8, w.z >> 8, w.w >> 8);
    const uint32_t sg = h2_add(__byte_perm(scg, H_1024, 0x5050 | B | ((B + 1) << 8)), H_M1024), sh = h2_add(__byte_perm(sch, H_1024, 0x5050 | B | ((B + 1) << 8)), H_M1024);
    const uint32_t kg = h2_mul(sg, H_M1024_M64), kh = h2_mul(sh, H_M1024_M64);
#pragma unroll
    for (int half = 0; half < 2; half++) {
        const uint32_t mask = half ? 0x00f000f0u : 0x000f000fu, under = half ? H_64 : H_1024;
        const uint32_t mg = half ? upper2(sg) : lower2(sg), mh = half ? upper2(sh) : lower2(sh), cg = half ? upper2(kg) : lower2(kg), ch = half ? upper2(kh) : lower2(kh);
        uint32_t* o = r + 8 * half;
        o[0] = h2_fma(and_or(w.x, mask, under), mg, cg);
        o[1] = h2_fma(and_or(w.y, mask, under), mh, ch);
        o[2] = h2_fma(and_or(v.x, mask, under), mg, cg);
        o[3] = h2_fma(and_or(v.y, mask, under), mh, ch);
        o[4] = h2_fma(and_or(w.z, mask, under), mg, cg);
        o[5] = h2_fma(and_or(w.w, mask, under), mh, ch);
        o[6] = h2_fma(and_or(v.z, mask, under), mg, cg);
        o[7] = h2_fma(and_or(v.w, mask, under), mh, ch);
    }
}
// The same of a Q6_K unit, from six code words; `sg`, `sh`: the words that hold the scales of its four 16-wide sub-blocks of rows g and g + 8, 128 added to every byte.
__device__ __forceinline__ void expand_q6k(const uint32_t* W, uint32_t sg, uint32_t sh, uint32_t (&r)[16]) {
#pragma unroll
    for (int G = 0; G < 2; G++) {
        const uint32_t w0 = W[3 * G], w1 = W[3 * G + 1], w2 = W[3 * G + 2];
        const uint32_t w3 = ((w0 << 6) & 0xc0c0c0c0u) | ((w1 << 4) & 0x30303030u) | ((w2 << 2) & 0x0c0c0c0cu);
        // bytes 4 (q - 32) + 128 under 1024: times scale / 4, less 288 scales
        const uint32_t r0 = (w0 & 0xfcfcfcfcu) ^ 0x80808080u, r1 = (w1 & 0xfcfcfcfcu) ^ 0x80808080u, r2 = (w2 & 0xfcfcfcfcu) ^ 0x80808080u, r3 = w3 ^ 0x80808080u;
        const uint32_t s0 = h2_add(__byte_perm(sg, H_1024, G ? 0x5352 : 0x5150), H_M1152), s1 = h2_add(__byte_perm(sh, H_1024, G ? 0x5352 : 0x5150), H_M1152);
        const uint32_t m0 = h2_mul(s0, H_QUARTER), m1 = h2_mul(s1, H_QUARTER), c0 = h2_mul(s0, H_M288), c1 = h2_mul(s1, H_M288);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t x0 = h ? r2 : r0, x1 = h ? r3 : r1;
            const uint32_t mg = h ? upper2(m0) : lower2(m0), mh = h ? upper2(m1) : lower2(m1), cg = h ? upper2(c0) : lower2(c0), ch = h ? upper2(c1) : lower2(c1);
            uint32_t* o = r + 8 * G + 4 * h;
            o[0] = h2_fma(__byte_perm(x0, H_1024, 0x5250), mg, cg);
            o[1] = h2_fma(__byte_perm(x1, H_1024, 0x5250), mh, ch);
            o[2] = h2_fma(__byte_perm(x0, H_1024, 0x5351), mg, cg);
            o[3] = h2_fma(__byte_perm(x1, H_1024, 0x5351), mh, ch);
        }
    }
}
// Columns 64 P .. of a Q6_K unit, `g`, `h`: the words that hold their sub-blocks' scales.
template <int P>
__device__ __forceinline__ void part_q6k(const uint8_t* sp, int lane, uint32_t g, uint32_t h, uint32_t (&r)[16]) {
    const uint4 u = reinterpret_cast<const uint4*>(sp)[(P * 3 / 2) * 32 + lane], v = reinterpret_cast<const uint4*>(sp)[(P * 3 / 2 + 1) * 32 + lane];
    const uint32_t lo[6] = {u.x, u.y, u.z, u.w, v.x, v.y}, hi[6] = {u.z, u.w, v.x, v.y, v.z, v.w};
    expand_q6k(P & 1 ? hi : lo, g ^ 0x80808080u, h ^ 0x80808080u, r);
}

// Which matrix a 16-row tile of the launch belongs to, and its first unit.
struct TileAt {
    const uint8_t* p;
    int s, local, ub;
};
__device__ __forceinline__ TileAt tile_at(const SgArgs& a, int tile, int kts) {
    TileAt r;
    r.s = 0;
    const uint8_t* w = a.seg[0].w;
    int t0 = 0, type = a.seg[0].type;
#pragma unroll
    for (int i = 1; i < 4; i++)
        if (i < a.nseg && tile >= a.seg[i].tile0) {
            r.s = i;
            w = a.seg[i].w;
            t0 = a.seg[i].tile0;
            type = a.seg[i].type;
        }
    r.local = tile - t0;
    r.ub = type == WT_Q6_K ? SG_UNIT_Q6K : SG_UNIT_Q4K;
    r.p = w + (size_t)r.local * kts * r.ub;
    return r;
}

// First item of CTA c of n; total * n fits 32 bits (checked by the launcher).
__device__ __forceinline__ int share(int c, int total, int n) { return (int)((unsigned)c * (unsigned)total / (unsigned)n); }

struct SgBars {
    uint64_t w_full[SG_W_SLOTS], w_free[SG_W_SLOTS];                              // an item's units
    uint64_t x_full[SG_X_SLOTS], x_free[SG_X_SLOTS], scale[SG_SCALE_SLOTS];       // its activations, their rows' scales
    uint64_t a_full[2];                                                           // the expanded weights of a team's item; their place is free when the sums are there
    uint64_t sum_full[2], sum_free[2];                                            // accumulators of even and odd items
    uint64_t out_full, out_free, last_full;                                       // sums of a group, of the CTA's last one
    uint64_t done[2];
    uint32_t tmem;
};

// The CTAs that hold blocks of a group: `n` from `first` on.  Of the first `ends` of them it is the last group, and the first `finish` of these finish it together, a share of its values
// each; the others (one that goes on with the next group, and those of a group in very many parts) only hand their sums over.  Finishers wait for CTAs before and behind them: there are
// eight at most, so that of a launch whose last CTAs are not resident yet up to seven hold an SM meanwhile.  21 launches in as many streams leave an SM free for those that are awaited;
// with more the waits may run out.
struct Parts {
    int first, n, ends, finish;
};
__device__ __forceinline__ Parts parts_of(int group, int kts, int total) {
    const unsigned n = gridDim.x, end = (unsigned)(group + 1) * kts;
    Parts p;
    p.first = (int)(((unsigned)group * kts * n + n - 1) / (unsigned)total);      // the largest c whose share does not begin behind the group's first item
    const int last = (int)((end * n - 1) / (unsigned)total);
    p.n = last - p.first + 1;
    p.ends = share(last + 1, total, n) == (int)end ? p.n : p.n - 1;
    p.finish = min(p.ends, 8);
    return p;
}
// A CTA's sums of its last group and of the one that its share begins in, as the others read them.  (With flags behind fences a launch took 1 us longer.)
__device__ __forceinline__ uint32_t* handed(const SgArgs& a, int cta, bool last) { return reinterpret_cast<uint32_t*>(a.ws) + (size_t)(2 * cta + last) * SG_WS_FLOATS; }
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// Quads of neighbouring rows [e0, e1) of group `group`, 32 to a row of x: the sums of this CTA (`out`, [row of x][128], complete when `ready` is), of the others of `p`, biases and what
// they are added to, stored by `threads` threads.  ITEMS quads of a thread and PARTS parts of each are under way at once; loads are not predicated (the last quad or part is read again)
// so that all of a round are.  Returns whether no wait ran out.
template <int ITEMS, int PARTS>
__device__ __forceinline__ bool finish_rows(const SgArgs& a, const float* out, int group, int kts, const Parts& p, int e0, int e1, int tid, int threads, uint64_t* ready) {
    const int lane = tid & 31, others = p.n - 1;
    const int row = ((e0 + lane) & 31) * 4, tile = group * SG_TILES + (row >> 4);      // the same in all rounds
    const bool glu = a.mode == 2;      // the up value of a gate is the next row
    const TileAt ta = tile_at(a, min(tile, a.tiles - 1), kts);
    const float* bias = a.seg[0].bias;
    int out_off = a.seg[0].out_off;
#pragma unroll
    for (int s = 1; s < 4; s++)
        if (s == ta.s) {
            bias = a.seg[s].bias;
            out_off = a.seg[s].out_off;
        }
    const int wrow = ta.local * 16 + (row & 15);
    float* o = a.out + ((out_off + wrow) >> glu);
    const bool wide = !(((uintptr_t)o | ((uintptr_t)a.ldo * 4)) & 15);
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (bias) b = make_float4(bias[wrow], bias[wrow + 1], bias[wrow + 2], bias[wrow + 3]);
#pragma unroll 1
    for (int base = e0 + tid - lane; base < e1; base += ITEMS * threads) {
        float4 y[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const int e = base + i * threads + lane;
            const float* r = o + (size_t)(e >> 5) * a.ldo;
            y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (a.mode == 1 && e < e1 && tile < a.tiles) {
                if (wide)
                    y[i] = __ldcg(reinterpret_cast<const float4*>(r));
                else
                    y[i] = make_float4(__ldcg(r), __ldcg(r + 1), __ldcg(r + 2), __ldcg(r + 3));
            }
        }
        // the others' last sums come when this CTA's do: asking for them before only gets in the way of what they write (at 64 rows 2 us of a launch)
        if (p.finish > 1 && ready) {
            if (!__all_sync(0xffffffffu, bar_wait(ready, 0))) return false;
            ready = nullptr;
        }
#pragma unroll 1
        for (int c0 = 0; c0 < others; c0 += PARTS) {
            uint4 v[ITEMS][PARTS];
            unsigned long long t0 = 0;
            for (;;) {
                bool there = true;
#pragma unroll
                for (int c = 0; c < PARTS; c++) {
                    const int part = p.first + min(c0 + c, others - 1), cta = part + (part >= (int)blockIdx.x);
                    const uint4* w = reinterpret_cast<const uint4*>(handed(a, cta, cta < p.first + p.ends));
#pragma unroll
                    for (int i = 0; i < ITEMS; i++) v[i][c] = ld_relaxed(w + min(base + i * threads + lane, e1 - 1));
                }
#pragma unroll
                for (int c = 0; c < PARTS; c++)
#pragma unroll
                    for (int i = 0; i < ITEMS; i++)
                        there &= base + i * threads + lane >= e1 || c0 + c >= others ||
                                 (v[i][c].x != HANDED_EMPTY && v[i][c].y != HANDED_EMPTY && v[i][c].z != HANDED_EMPTY && v[i][c].w != HANDED_EMPTY);
                if (__all_sync(0xffffffffu, there)) break;
                const unsigned long long t = __shfl_sync(0xffffffffu, now_ns(), 0);
                if (t0 == 0) t0 = t;
                if (t - t0 > SG_WAIT_NS) return false;
            }
#pragma unroll
            for (int c = 0; c < PARTS; c++)
                if (c0 + c < others) {
                    const int part = p.first + c0 + c, cta = part + (part >= (int)blockIdx.x);
                    uint4* w = reinterpret_cast<uint4*>(handed(a, cta, cta < p.first + p.ends));
#pragma unroll
                    for (int i = 0; i < ITEMS; i++) {
                        const int e = base + i * threads + lane;
                        if (e < e1) st_relaxed(w + e, make_uint4(HANDED_EMPTY, HANDED_EMPTY, HANDED_EMPTY, HANDED_EMPTY));
                        y[i] = add4(y[i], make_float4(__uint_as_float(v[i][c].x), __uint_as_float(v[i][c].y), __uint_as_float(v[i][c].z), __uint_as_float(v[i][c].w)));
                    }
                }
        }
        if (ready) {
            if (!__all_sync(0xffffffffu, bar_wait(ready, 0))) return false;
            ready = nullptr;
        }
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const int e = base + i * threads + lane;
            if (e < e1 && tile < a.tiles) {
                const float4 v = add4(add4(y[i], *reinterpret_cast<const float4*>(out + 4 * e)), b);
                float* r = o + (size_t)(e >> 5) * a.ldo;
                if (glu) {
                    r[0] = glu_act(v.x, v.y, a.act, a.alpha, a.limit);
                    r[1] = glu_act(v.z, v.w, a.act, a.alpha, a.limit);
                } else if (wide) {
                    *reinterpret_cast<float4*>(r) = v;
                } else {
                    r[0] = v.x;
                    r[1] = v.y;
                    r[2] = v.z;
                    r[3] = v.w;
                }
            }
        }
    }
    return true;
}

template <int NT>
__global__ void __launch_bounds__(SG_THREADS, 1) gemm_sk_kernel(const __grid_constant__ SgArgs a) {
    constexpr int N = 16 * NT, X_BYTES = N * SG_ROW, X_SLOT = (X_BYTES + 1023) & ~1023, CHUNK = NT * SG_CHUNK;
    constexpr bool ONE_MINS = NT == 4;             // sums of the minima: one place instead of two, where tensor memory is full
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) SgBars bars;
    __shared__ Parts last_parts;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kts = a.k >> 8, total = (a.tiles + SG_TILES - 1) / SG_TILES * kts;
    const int lo = share(blockIdx.x, total, gridDim.x), n_items = share(blockIdx.x + 1, total, gridDim.x) - lo;
    const int group0 = lo / kts, kb_lo = lo - group0 * kts;
    const int XS = a.x_slots, R = a.ring;
    uint8_t* x_ring = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    float2* dbuf = reinterpret_cast<float2*>(x_ring + XS * X_SLOT);            // [slot][128]
    float* scales = reinterpret_cast<float*>(dbuf + SG_D_SLOTS * 128);         // [slot][N]
    float* out = scales + SG_SCALE_SLOTS * N;                                  // [row of x][128]
    uint8_t* w_ring = reinterpret_cast<uint8_t*>(out + N * 128);               // [slot][tile]
    if (threadIdx.x == 0) {
        for (int i = 0; i < R; i++) {
            mbar_init(&bars.w_full[i], SG_TILES);
            mbar_init(&bars.w_free[i], SG_TILES);
        }
        for (int i = 0; i < XS; i++) {
            mbar_init(&bars.x_full[i], 1);
            mbar_init(&bars.x_free[i], 1);
        }
        for (int i = 0; i < SG_SCALE_SLOTS; i++) mbar_init(&bars.scale[i], 1);
        for (int i = 0; i < 2; i++) {
            mbar_init(&bars.a_full[i], SG_TILES);
            mbar_init(&bars.sum_full[i], 1);
            mbar_init(&bars.sum_free[i], SG_SUM);
            mbar_init(&bars.done[i], 1);
        }
        mbar_init(&bars.out_full, SG_SUM);
        mbar_init(&bars.out_free, SG_FINISH);
        mbar_init(&bars.last_full, SG_SUM);
        last_parts = parts_of((lo + n_items - 1) / kts, kts, total);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_launch();
    bool alive = true;      // false: a wait ran out
    auto wait = [&](uint64_t* bar, uint32_t parity) { return alive = __all_sync(0xffffffffu, bar_wait(bar, parity)) != 0; };

    if (warp < SG_EXPAND) {
        const int quad = warp & 3, team = warp >> 3, tig = 2 * quad + ((warp >> 2) & 1);      // warp & 3 gives the TMEM lanes it reaches
        __syncthreads();      // barriers and tensor memory
        tc_fence_after();
        const uint32_t a_cols = bars.tmem + ((uint32_t)(quad * 32 + 16 * ((warp >> 2) & 1)) << 16) + team * SG_A_COLS;
        const int g = lane >> 2, t = lane & 3, row = tig * 16 + g;
        int slot = team, kb = kb_lo + team, tile = group0 * SG_TILES + tig;
        uint32_t turn = 0;
        bool fresh = true, mine = false, q6 = false;
        for (int i = team; i < n_items; i += 2) {
            if (kb >= kts) {
                do {
                    kb -= kts;
                    tile += SG_TILES;
                } while (kb >= kts);
                fresh = true;
            }
            if (fresh) {
                mine = tile < a.tiles;
                q6 = mine && tile_at(a, tile, kts).ub == SG_UNIT_Q6K;
                fresh = false;
            }
            if (!wait(&bars.w_full[slot], turn)) break;
            const uint8_t* sp = w_ring + (size_t)(slot * SG_TILES + tig) * a.slot_bytes;
            uint4 sg, sh;
            float2 dg, dh;
            uint32_t r[16];
            if (q6) {
                sg = reinterpret_cast<const uint4*>(sp + 3072)[g];
                sh = reinterpret_cast<const uint4*>(sp + 3072)[g + 8];
                dg = make_float2(__half2float(reinterpret_cast<const __half*>(sp + 3328)[g]), 0.f);
                dh = make_float2(__half2float(reinterpret_cast<const __half*>(sp + 3328)[g + 8]), 0.f);
                part_q6k<0>(sp, lane, sg.x, sh.x, r);
            } else {
                sg = reinterpret_cast<const uint4*>(sp + 2048)[g];
                sh = reinterpret_cast<const uint4*>(sp + 2048)[g + 8];
                dg = __half22float2(reinterpret_cast<const __half2*>(sp + 2304)[g]);
                dh = __half22float2(reinterpret_cast<const __half2*>(sp + 2304)[g + 8]);
                expand_q4k<0>(reinterpret_cast<const uint4*>(sp)[lane], sg.x, sh.x, r);
            }
            if (i > 1) {
                if (!wait(&bars.sum_full[team], ((i >> 1) - 1) & 1)) break;
                tc_fence_after();
            }
            tmem_st_16x128_x8(a_cols, r);
            uint32_t m0 = 0, m1 = 0;      // minima 2 t, 2 t + 1 of both rows
            if (q6) {
                part_q6k<1>(sp, lane, sg.y, sh.y, r);
                tmem_st_16x128_x8(a_cols + 32, r);
                part_q6k<2>(sp, lane, sg.z, sh.z, r);
                tmem_st_16x128_x8(a_cols + 64, r);
                part_q6k<3>(sp, lane, sg.w, sh.w, r);
            } else {
                expand_q4k<2>(reinterpret_cast<const uint4*>(sp)[32 + lane], sg.x, sh.x, r);
                tmem_st_16x128_x8(a_cols + 32, r);
                expand_q4k<0>(reinterpret_cast<const uint4*>(sp)[64 + lane], sg.y, sh.y, r);
                tmem_st_16x128_x8(a_cols + 64, r);
                expand_q4k<2>(reinterpret_cast<const uint4*>(sp)[96 + lane], sg.y, sh.y, r);
                const uint32_t wg = (t < 2 ? sg.z : sg.w) >> (16 * (t & 1)), wh = (t < 2 ? sh.z : sh.w) >> (16 * (t & 1));
                m0 = h2_add(__byte_perm(wg, H_1024, 0x5150), H_M1024);
                m1 = h2_add(__byte_perm(wh, H_1024, 0x5150), H_M1024);
            }
            __syncwarp();      // every lane has its part of the unit
            if (lane == 0) mbar_arrive(&bars.w_free[slot]);
            tmem_st_16x128_x8(a_cols + 96, r);
            tmem_st_16x128_x2(a_cols + 128, m0, m1, m0, m1);      // for the upper and again for the lower parts of the sums of 32
            if (t == 0) {
                // the sums of the item that had the slot before are taken: the products of the one two items ago, which have ended, waited for those of two more before
                float2* my_d = dbuf + (i & (SG_D_SLOTS - 1)) * 128 + row;
                my_d[0] = dg;
                my_d[8] = dh;
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.a_full[team]);
            slot += 2;
            if (slot >= R) {
                slot -= R;
                turn ^= 1;
            }
            kb += 2;
        }
        // nothing more to expand: all sixteen warps finish the last group
        pdl_wait();
        const int last = (lo + n_items - 1) / kts, quads = a.nb * 32;
        const Parts p = last_parts;
        if (!alive) {
        } else if (p.finish > 1) {
            const int j = blockIdx.x - p.first;
            if (j < p.finish)
                alive = finish_rows<1, 4>(a, out, last, kts, p, share(j, quads, p.finish), share(j + 1, quads, p.finish), threadIdx.x, SG_EXPAND * 32, &bars.last_full);
        } else {
            alive = finish_rows<4, 1>(a, out, last, kts, p, 0, quads, threadIdx.x, SG_EXPAND * 32, &bars.last_full);
        }
    } else if (warp < SG_MMA) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 136;");
        __syncthreads();
        tc_fence_after();
        const int quad = warp & 3, row = quad * 32 + lane;
        const uint32_t cols = bars.tmem + ((uint32_t)(quad * 32) << 16) + 2 * SG_A_COLS;
        int group = group0, kb0 = kb_lo;
        for (int i = 0; i < n_items; group++, kb0 = 0) {
            const int n_seg = min(n_items - i, kts - kb0);
            f2 sum[N / 2];
#pragma unroll
            for (int c = 0; c < N / 2; c++) sum[c] = 0ull;
            for (const int end = i + n_seg; i < end; i++) {
                const int buf = i & 1;
                if (!wait(&bars.scale[i & (SG_SCALE_SLOTS - 1)], (i / SG_SCALE_SLOTS) & 1) || !wait(&bars.sum_full[buf], (i >> 1) & 1)) break;
                tc_fence_after();
                const float2 d = dbuf[(i & (SG_D_SLOTS - 1)) * 128 + row];
                const f2 d2 = pack2(d.x, d.x), m2 = pack2(-d.y, -d.y);
                const ulonglong2* sx = reinterpret_cast<const ulonglong2*>(scales + (i & (SG_SCALE_SLOTS - 1)) * N);
                const uint32_t at = cols + buf * N, at_m = cols + 2 * N + (ONE_MINS ? 0 : buf * N);
#pragma unroll
                for (int c = 0; c < NT; c++) {
                    uint32_t v[16], m[16];
                    tmem_ld16(at + 16 * c, v);
                    tmem_ld16(at_m + 16 * c, m);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (c == NT - 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bars.sum_free[buf]);
                    }
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const ulonglong2 s = sx[4 * c + (j >> 1)];
                        sum[8 * c + j] = fma2(s.x, fma2(m2, pack2u(m[2 * j], m[2 * j + 1]), mul2(d2, pack2u(v[2 * j], v[2 * j + 1]))), sum[8 * c + j]);
                        sum[8 * c + j + 1] = fma2(s.y, fma2(m2, pack2u(m[2 * j + 2], m[2 * j + 3]), mul2(d2, pack2u(v[2 * j + 2], v[2 * j + 3]))), sum[8 * c + j + 1]);
                    }
                }
            }
            if (!alive) break;
            // the rows are finished by other warps: here the stores and their fence took 6000 cycles, in which nothing moved
            const bool last = i == n_items;
            if (group > group0 && !wait(&bars.out_free, (group - group0 - 1) & 1)) break;
            const auto hand_over = [&] {      // all but what this CTA finishes itself
                const Parts p = last_parts;
                if (!last || p.ends < 2) return;
                uint32_t* w = handed(a, blockIdx.x, true) + row;
                const int j = blockIdx.x - p.first, quad = row >> 2;
                const int e0 = j < p.finish ? share(j, a.nb * 32, p.finish) : 0, e1 = j < p.finish ? share(j + 1, a.nb * 32, p.finish) : 0;
#pragma unroll
                for (int c = 0; c < N; c++) {
                    const float2 v = unpack2(sum[c >> 1]);
                    if (c < a.nb && (c * 32 + quad < e0 || c * 32 + quad >= e1)) st_relaxed(w + c * 128, handed_bits(c & 1 ? v.y : v.x));
                }
            };
            // the others wait for it, so it goes first; but 64 stores in a row hold up the sums for this CTA's own threads (a layer at 64 rows: 93 us, 87 after them; 65 and 66 at 32)
            if (NT < 4) hand_over();
#pragma unroll
            for (int c = 0; c < N / 2; c++) {
                const float2 v = unpack2(sum[c]);
                out[(2 * c) * 128 + row] = v.x;
                out[(2 * c + 1) * 128 + row] = v.y;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(last ? &bars.last_full : &bars.out_full);
            if (NT == 4) hand_over();
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == SG_MMA) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&bars.tmem)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
            tc_fence_before();
        }
        __syncthreads();
        tc_fence_after();
        if (warp < SG_LOAD_X) {
            // products of every second item: with one warp for all, its waits and the issue of 17 instructions (1250 cycles an item) were the slowest part
            const int par = warp - SG_MMA;
            const uint32_t tmem = __shfl_sync(0xffffffffu, bars.tmem, 0);
            const uint32_t d = tmem + 2 * SG_A_COLS + par * N, dm = tmem + 2 * SG_A_COLS + 2 * N + (ONE_MINS ? 0 : par * N), at = tmem + par * SG_A_COLS;
            const uint64_t x_desc = umma_desc(x_ring), s_desc = desc_cells(smem_u32(x_ring) + N * 512, N * 16);
            int s = par;
            uint32_t turn = 0, lap = 0;
            for (int i = par; i < n_items; i += 2, lap ^= 1) {
                if (!wait(&bars.x_full[s], turn) || (i > 1 && !wait(&bars.sum_free[par], lap ^ 1)) || !wait(&bars.a_full[par], lap)) break;
                tc_fence_after();
                const uint64_t x0 = (uint64_t)((s * X_SLOT) >> 4), xd = x_desc + x0;
                if (elect()) {
#pragma unroll
                    for (int c = 0; c < 16; c++) mma_ts(d, at + c * 8, xd + (uint64_t)(((c >> 2) * N * 128 + (c & 3) * 32) >> 4), sg_idesc(N), c > 0);
                }
                __syncwarp();
                if (ONE_MINS && i > 0) {
                    if (!wait(&bars.sum_free[par ^ 1], ((i - 1) >> 1) & 1)) break;
                    tc_fence_after();
                }
                if (elect()) {
                    mma_ts(dm, at + 128, s_desc + x0, sg_idesc(N), 0);
                    umma_commit(&bars.sum_full[par]);
                    umma_commit(&bars.x_free[s]);
                }
                __syncwarp();
                s += 2;
                if (s >= XS) {
                    s -= XS;
                    turn ^= 1;
                }
            }
            if (!alive) {      // what is under way ends before the CTA leaves
                if (elect()) umma_commit(&bars.done[par]);
                bar_wait(&bars.done[par], 0);
            }
        } else if (warp == SG_LOAD_X) {
            pdl_wait();
            int kb = kb_lo, s = 0, i = 0;
            uint32_t turn = 0;
            for (; i < n_items; i++) {
                if (i >= XS && !wait(&bars.x_free[s], turn ^ 1)) break;
                const int q = i & (SG_SCALE_SLOTS - 1);      // free: the accumulators of two items before the one that had the slot of x were
                if (lane == 0) {
                    const uint8_t* src = a.x + (size_t)kb * CHUNK;
                    mbar_expect_tx(&bars.x_full[s], X_BYTES);
                    bulk_copy(smem_u32(x_ring + s * X_SLOT), src, X_BYTES, &bars.x_full[s]);
                    mbar_expect_tx(&bars.scale[q], N * 4);
                    bulk_copy(smem_u32(scales + q * N), src + X_BYTES, N * 4, &bars.scale[q]);
                }
                __syncwarp();
                if (++kb == kts) kb = 0;
                if (++s == XS) {
                    s = 0;
                    turn ^= 1;
                }
            }
            if (!alive)      // what is under way ends before the CTA leaves
                for (int j = i - XS; j < i; j++) {
                    bar_wait(&bars.x_full[j % XS], (j / XS) & 1);
                    bar_wait(&bars.scale[j & (SG_SCALE_SLOTS - 1)], (j / SG_SCALE_SLOTS) & 1);
                }
        } else if (warp < SG_LAST) {
            // units of every second item: lane i copies the one of the group's i-th tile (eight copies take a warp 1000 cycles)
            uint64_t policy;
            asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
            const int par = warp - SG_LOAD_W;
            int kb = kb_lo + par, tile = group0 * SG_TILES + lane, slot = par, i = par;
            uint32_t turn = 0, bytes = 0;
            const uint8_t* p = nullptr;
            bool fresh = true;
            for (; i < n_items; i += 2) {
                if (kb >= kts) {
                    do {
                        kb -= kts;
                        tile += SG_TILES;
                    } while (kb >= kts);
                    fresh = true;
                }
                if (fresh) {
                    bytes = 0;
                    if (lane < SG_TILES && tile < a.tiles) {
                        const TileAt ta = tile_at(a, tile, kts);
                        bytes = ta.ub;
                        p = ta.p + (size_t)kb * bytes;
                    }
                    fresh = false;
                }
                if (i >= R && !wait(&bars.w_free[slot], turn ^ 1)) break;
                if (bytes) {
                    mbar_expect_tx(&bars.w_full[slot], bytes);
                    bulk_copy(smem_u32(w_ring + (size_t)(slot * SG_TILES + lane) * a.slot_bytes), p, bytes, &bars.w_full[slot], policy);
                    p += 2 * bytes;
                } else if (lane < SG_TILES) {
                    mbar_arrive(&bars.w_full[slot]);
                }
                __syncwarp();
                slot += 2;
                if (slot >= R) {
                    slot -= R;
                    turn ^= 1;
                }
                kb += 2;
            }
            if (!alive)      // what is under way ends before the CTA leaves
                for (int j = max(par, i - (R & ~1)); j < i; j += 2) bar_wait(&bars.w_full[j % R], (j / R) & 1);
        } else {
            pdl_wait();
            int kb0 = kb_lo;
            const int last = (lo + n_items - 1) / kts, tid = threadIdx.x - SG_LAST * 32;
            for (int g = group0; g < last; g++, kb0 = 0) {
                if (!wait(&bars.out_full, (g - group0) & 1)) break;
                if (kb0) {
                    uint4* w = reinterpret_cast<uint4*>(handed(a, blockIdx.x, false));
                    for (int e = tid; e < a.nb * 32; e += SG_FINISH * 32) {
                        const float4 v = *reinterpret_cast<const float4*>(out + 4 * e);
                        st_relaxed(w + e, make_uint4(handed_bits(v.x), handed_bits(v.y), handed_bits(v.z), handed_bits(v.w)));
                    }
                } else {
                    finish_rows<1, 1>(a, out, g, kts, Parts{(int)blockIdx.x, 1, 1, 1}, 0, a.nb * 32, tid, SG_FINISH * 32, nullptr);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars.out_free);
            }
        }
    }
    if (!alive && lane == 0) *(volatile int*)a.status = KS_TIMEOUT;
    tc_fence_before();
    __syncthreads();
    if (warp == SG_MMA) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(bars.tmem));
    }
}

// One warp per (row, 256-block): eight columns per lane.  A row that is normalised belongs to one CTA (its sum of squares is needed first).
// Rows nb .. 16 ceil(nb / 16) - 1 are written as zeros.
template <bool BF16>
__device__ __forceinline__ void load8(const void* x, size_t at, float (&v)[8]) {
    if (BF16) {
        const uint4 u = __ldcg(reinterpret_cast<const uint4*>((const __nv_bfloat16*)x + at));
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    } else {
        const float4* p = reinterpret_cast<const float4*>((const float*)x + at);
        const float4 u0 = __ldcg(p), u1 = __ldcg(p + 1);
        v[0] = u0.x; v[1] = u0.y; v[2] = u0.z; v[3] = u0.w; v[4] = u1.x; v[5] = u1.y; v[6] = u1.z; v[7] = u1.w;
    }
}

constexpr int R16_WARPS = 8, R16_KEEP = 8;      // blocks that a warp keeps in registers between the sum of squares and the stores

template <bool BF16>
__global__ void __launch_bounds__(R16_WARPS * 32) rows16_kernel(const __grid_constant__ Rows16Args a, int nb) {
    __shared__ float ssq[R16_WARPS];
    pdl_launch();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = blockIdx.x, nkb = a.k >> 8, n = gridDim.x;
    const int b0 = blockIdx.y * R16_WARPS + warp, step = gridDim.y * R16_WARPS;
    const bool pad = row >= nb;
    if (!a.norm_w) {
        for (int blk = b0; blk < nkb; blk += step) {
            float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (!pad) load8<BF16>(a.x, (size_t)row * a.ldx + blk * 256 + lane * 8, v);
            store_block16(a.out, n, row, blk, lane, v);
        }
        return;
    }
    float v[R16_KEEP][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < R16_KEEP; i++) {
        const int blk = warp + i * R16_WARPS;
        if (blk < nkb && !pad) load8<BF16>(a.x, (size_t)row * a.ldx + blk * 256 + lane * 8, v[i]);
        else
#pragma unroll
            for (int j = 0; j < 8; j++) v[i][j] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < R16_KEEP; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) ss += v[i][j] * v[i][j];
    ss = warp_sum(ss);
    if (lane == 0) ssq[warp] = ss;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < R16_WARPS; i++) s += ssq[i];
    const float rstd = rsqrtf(s / (float)a.k + a.eps);
#pragma unroll
    for (int i = 0; i < R16_KEEP; i++) {
        const int blk = warp + i * R16_WARPS;
        if (blk >= nkb) break;
        const float4* n4 = reinterpret_cast<const float4*>(a.norm_w + blk * 256 + lane * 8);
        const float4 n0 = n4[0], n1 = n4[1];
        const float w[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
#pragma unroll
        for (int j = 0; j < 8; j++) v[i][j] *= rstd * w[j];
        store_block16(a.out, n, row, blk, lane, v[i]);
    }
}

int sms() {
    static int n[64] = {};
    int d = 0;
    cudaGetDevice(&d);
    d &= 63;
    if (!n[d]) cudaDeviceGetAttribute(&n[d], cudaDevAttrMultiProcessorCount, d);
    return n[d];
}

int go(const void* fn, dim3 grid, dim3 block, size_t smem, void** args, cudaStream_t st, int pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace

// Bytes of the activation chunks of nb rows of length k.
B2_API long long b2_rows16_bytes(int nb, int k) { return (long long)(k >> 8) * ((nb + 15) >> 4) * SG_CHUNK; }

// Rows in the order that b2_gemm_sk reads.  k a multiple of 256 (at most 16384 with a norm), x and out 16-byte aligned, ldx a multiple of 8 (fp32: of 4).
B2_API int b2_rows16(const Rows16Args* in, int nb, int pdl, cudaStream_t st) {
    Rows16Args a = *in;
    if (nb < 1 || nb > SG_MAX_ROWS || a.k < 256 || (a.k & 255) || !a.x || !a.out || (((uintptr_t)a.x | (uintptr_t)a.out | (uintptr_t)a.norm_w) & 15) ||
        (a.ldx & (a.bf16 ? 7 : 3)))
        return (int)cudaErrorInvalidValue;
    if (a.norm_w && (a.k >> 8) > R16_WARPS * R16_KEEP) return (int)cudaErrorNotSupported;
    const int nkb = a.k >> 8, rows = (nb + 15) & ~15;
    void* args[] = {&a, &nb};
    const dim3 grid(rows, a.norm_w ? 1 : (nkb + R16_WARPS - 1) / R16_WARPS);
    return go(a.bf16 ? (const void*)rows16_kernel<true> : (const void*)rows16_kernel<false>, grid, dim3(R16_WARPS * 32), 0, args, st, pdl);
}

// Floats of the workspace of b2_gemm_sk, every byte of which is 255 before the first launch and whenever a launch has ended (unless a wait ran out).
B2_API long long b2_gemm_sk_ws() { return 2ll * SG_CTAS * SG_WS_FLOATS; }

// y = W x for 1..64 rows in the chunks of b2_rows16, up to four matrices of one row length.  Returns a cudaError_t value.
B2_API int b2_gemm_sk(const SgArgs* in, int max_ctas, int pdl, cudaStream_t st) {
    SgArgs a = *in;
    if (a.nseg < 1 || a.nseg > 4 || a.nb < 1 || a.nb > SG_MAX_ROWS || a.k < 256 || (a.k & 255) || !a.x || ((uintptr_t)a.x & 15) || !a.out || !a.ws || ((uintptr_t)a.ws & 15) || !a.status ||
        a.mode < 0 || a.mode > 2)
        return (int)cudaErrorInvalidValue;
    int slot = 0, tiles = 0;
    for (int s = 0; s < a.nseg; s++) {
        SgSeg& g = a.seg[s];
        if ((g.type != WT_Q4_K && g.type != WT_Q6_K) || g.n <= 0 || (g.n & 15) || ((uintptr_t)g.w & 15) || (a.mode == 2 && (g.out_off & 1))) return (int)cudaErrorInvalidValue;
        g.tile0 = tiles;
        tiles += g.n >> 4;
        slot = slot > (g.type == WT_Q6_K ? SG_UNIT_Q6K : SG_UNIT_Q4K) ? slot : (g.type == WT_Q6_K ? SG_UNIT_Q6K : SG_UNIT_Q4K);
    }
    const int nt = (a.nb + 15) >> 4, rows = 16 * nt;
    a.tiles = tiles;
    a.slot_bytes = slot;
    const size_t chunk = (size_t)((rows * SG_ROW + 1023) & ~1023);
    const size_t fixed = 1024 + SG_D_SLOTS * 128 * 8 + SG_SCALE_SLOTS * rows * 4 + rows * 512, item = (size_t)SG_TILES * slot;
    // Four chunks of activations where at least four items fit beside them, else two (32 rows and fewer: six or eight items beside four chunks; 64: four or six beside two).  Both
    // rings are even, so that a slot always belongs to even or to odd items: the warps that fill or use it wait for every phase of its barriers, as the parity of a phase demands.
    a.x_slots = fixed + 4 * chunk + 4 * item <= SG_MAX_SMEM ? 4 : 2;
    const size_t slots = (SG_MAX_SMEM - fixed - a.x_slots * chunk) / item;
    a.ring = (slots < SG_W_SLOTS ? (int)slots : SG_W_SLOTS) & ~1;
    const size_t smem = fixed + a.x_slots * chunk + a.ring * item;
    const void* fn = nt == 1 ? (const void*)gemm_sk_kernel<1> : nt == 2 ? (const void*)gemm_sk_kernel<2> : nt == 3 ? (const void*)gemm_sk_kernel<3> : (const void*)gemm_sk_kernel<4>;
    static PerDeviceOnce once[SG_MAX_NT];
    if (once[nt - 1].first()) {
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SG_MAX_SMEM);
        if (e != cudaSuccess) return (int)e;
    }
    const int total = (tiles + SG_TILES - 1) / SG_TILES * (a.k >> 8);
    if (total >= 1 << 23) return (int)cudaErrorNotSupported;
    // one CTA per SM: all are resident, so waits on other CTAs end.  No more of them than give every CTA as many items as the fullest has.
    int grid = total < sms() ? total : sms();
    if (grid > SG_CTAS) grid = SG_CTAS;            // CTAs that the workspace holds two parts of
    if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
    const int most = (total + grid - 1) / grid;
    grid = (total + most - 1) / most;
    void* args[] = {&a};
    return go(fn, dim3((unsigned)grid), dim3(SG_THREADS), smem, args, st, pdl);
}
