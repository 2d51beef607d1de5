// Product of 1..32 rows with unit-ordered Q4_K / Q6_K matrices (the layout of gemv_sk.cu) in 16-bit activations, sm_100a.
//
// Decode steps of several sequences and short passes (drafted tokens, ends of prompts) multiply a few rows with matrices that stream from HBM once.
// The bound is that stream, so nothing else may cost more than it:
//   * Activations.  b2_rows16 turns fp32 or bf16 rows (optionally RMS-normalised) into f16 values with one power-of-two scale per row and 256-block, stored in the
//     order in which the lanes of a warp load tensor-core B fragments: [256-block][8 rows][...].  One 256-block of all rows is one contiguous chunk of 4384 bytes per
//     eight rows that a producer warp copies into shared memory once per CTA (cp.async.bulk, a ring of chunks); all 16 warps of the CTA read it with
//     conflict-free 16-byte loads.  (The int8 form that this replaces gathered its operand as 4-byte words through L1: per unit of 2.4 KB a warp fetched 8 KB in
//     sectors of 16 used bytes at 32 rows, and a launch took 69 us where its weights stream in 10.)
//   * Weights.  Each warp owns one 16-row tile per group of 16 tiles and streams its units through a cp.async ring of its own, requested before the grid-dependency wait.
//     Codes become f16 A fragments in registers: a 4-bit code under the exponent of 1024 and one fused multiply-add give code x 6-bit scale exactly (at most 945); of
//     Q6_K code x scale is rounded once to 11 bits.  mma.sync m16n8k16 sums a 256-block in fp32; the block's d and the rows' scales are applied to the sums, and the
//     Q4_K minima are one more mma per block, whose B fragment holds the rows' sums of 32 in two f16 parts.
//     So neither operand is rounded to fewer bits than the f16 activation keeps (2^-12 of a block's largest value at worst, against 2^-8 of the int8 form and
//     2^-9 of products on bf16 copies): relative error of a product against 64 bits 2.1e-4 (Q4_K) and 2.6e-4 (Q6_K), int8 form 7e-3.
//   * Work.  The launch's (group, 256-block) items are dealt out in equal contiguous shares, one CTA per SM; a group that is split between CTAs is finished by the CTA
//     that holds its first block, which adds the others' sums in a fixed order (workspace + flag per warp, bounded wait), as in gemv_sk.cu.
#include "pass_args.cuh"

namespace {

constexpr int SG_WARPS = 16;                        // consumer warps = row tiles of a group
constexpr int SG_THREADS = (SG_WARPS + 1) * 32;     // and the producer warp
constexpr int SG_UNIT_Q4K = 2368, SG_UNIT_Q6K = 3360;
constexpr int SG_FRAG = 4096, SG_SUMS = 256, SG_CHUNK = SG_FRAG + SG_SUMS + 32;      // bytes per 256-block and eight rows: values, sums of 32, scales
constexpr int SG_WS_FLOATS = 16 * 32;
constexpr int SG_MAX_SMEM = 225 * 1024;
constexpr unsigned long long SG_WAIT_NS = 1000000000ull;

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory"); }
__device__ __forceinline__ void bar_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory"); }
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity) {      // bounded: about a second
    for (int i = 0; i < (1 << 22); i++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(smem_addr(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if (i > 128) __nanosleep(100);
    }
    return false;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) { asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, uint64_t policy) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy) : "memory");
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
__device__ __forceinline__ void mma16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// f16x2 constants: 1024 under a code, and what takes it (times a scale) away again
constexpr uint32_t H_1024 = 0x64006400u, H_M1024 = 0xE400E400u, H_M64 = 0xD400D400u, H_16TH = 0x2C002C00u, H_M1152 = 0xE480E480u, H_QUARTER = 0x34003400u,
                   H_M288 = 0xDC80DC80u;

// byte b of w (0..255) twice as f16x2, 1024 added
__device__ __forceinline__ uint32_t byte_h2(uint32_t w, int b) { return __byte_perm(w, H_1024, 0x5050 | b | (b << 8)); }

}  // namespace

namespace {

// Sums of one unit (16 rows x 256 columns) with all rows of the chunk.  `xc`: the chunk in shared memory.
template <int NT>
__device__ __forceinline__ void unit16_q4k(const uint8_t* sp, const uint8_t* xc, int lane, float (&facc)[NT][4]) {
    const int g = lane >> 2, t = lane & 3;
    const uint4 sg = reinterpret_cast<const uint4*>(sp + 2048)[g], sh = reinterpret_cast<const uint4*>(sp + 2048)[g + 8];
    const float2 dg = __half22float2(reinterpret_cast<const __half2*>(sp + 2304)[g]);
    const float2 dh = __half22float2(reinterpret_cast<const __half2*>(sp + 2304)[g + 8]);
    const uint4* xf = reinterpret_cast<const uint4*>(xc) + lane;
    float acc[NT == 1 ? 2 : NT][4];      // one group of rows: two chains of dependent products
#pragma unroll
    for (int n = 0; n < (NT == 1 ? 2 : NT); n++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[n][i] = 0.f;
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const uint4 w = reinterpret_cast<const uint4*>(sp)[p * 32 + lane];
        const uint4 v = make_uint4(w.x >> 8, w.y >> 8, w.z >> 8, w.w >> 8);
        const uint32_t scg = p < 2 ? sg.x : sg.y, sch = p < 2 ? sh.x : sh.y;
#pragma unroll
        for (int half = 0; half < 2; half++) {      // low nibbles: sub-block 2p, high nibbles: 2p + 1
            const int b = ((2 * p) & 3) + half;
            const uint32_t mask = half ? 0x00f000f0u : 0x000f000fu;
            const uint32_t s0 = h2_add(byte_h2(scg, b), H_M1024), s1 = h2_add(byte_h2(sch, b), H_M1024);
            const uint32_t mg = half ? h2_mul(s0, H_16TH) : s0, mh = half ? h2_mul(s1, H_16TH) : s1;
            const uint32_t cg = h2_mul(s0, half ? H_M64 : H_M1024), ch = h2_mul(s1, half ? H_M64 : H_M1024);
            const uint32_t a0 = h2_fma((w.x & mask) | H_1024, mg, cg), a1 = h2_fma((w.y & mask) | H_1024, mh, ch);
            const uint32_t a2 = h2_fma((v.x & mask) | H_1024, mg, cg), a3 = h2_fma((v.y & mask) | H_1024, mh, ch);
            const uint32_t e0 = h2_fma((w.z & mask) | H_1024, mg, cg), e1 = h2_fma((w.w & mask) | H_1024, mh, ch);
            const uint32_t e2 = h2_fma((v.z & mask) | H_1024, mg, cg), e3 = h2_fma((v.w & mask) | H_1024, mh, ch);
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const uint4 bv = xf[n * (SG_FRAG / 16) + (2 * p + half) * 32];
                mma16(acc[n], a0, a1, a2, a3, bv.x, bv.y);
                mma16(acc[NT == 1 ? 1 : n], e0, e1, e2, e3, bv.z, bv.w);
            }
        }
    }
    // minima 2t, 2t + 1 of both rows; k slots 0..7 meet the upper, 8..15 the lower parts of the sums of 32
    const uint32_t wg = (t < 2 ? sg.z : sg.w) >> (16 * (t & 1)), wh = (t < 2 ? sh.z : sh.w) >> (16 * (t & 1));
    const uint32_t m0 = h2_add(__byte_perm(wg, H_1024, 0x5150), H_M1024), m1 = h2_add(__byte_perm(wh, H_1024, 0x5150), H_M1024);
    const uint2* xs = reinterpret_cast<const uint2*>(xc + NT * SG_FRAG) + lane;
    const float2* xd = reinterpret_cast<const float2*>(xc + NT * (SG_FRAG + SG_SUMS)) + t;
#pragma unroll
    for (int n = 0; n < NT; n++) {
        const uint2 bv = xs[n * 32];
        float am[4] = {0.f, 0.f, 0.f, 0.f};
        mma16(am, m0, m1, m0, m1, bv.x, bv.y);
        const float2 d = xd[n * 4];
        if (NT == 1) {
#pragma unroll
            for (int i = 0; i < 4; i++) acc[0][i] += acc[1][i];
        }
        facc[n][0] += d.x * (dg.x * acc[n][0] - dg.y * am[0]);
        facc[n][1] += d.y * (dg.x * acc[n][1] - dg.y * am[1]);
        facc[n][2] += d.x * (dh.x * acc[n][2] - dh.y * am[2]);
        facc[n][3] += d.y * (dh.x * acc[n][3] - dh.y * am[3]);
    }
}

template <int NT>
__device__ __forceinline__ void unit16_q6k(const uint8_t* sp, const uint8_t* xc, int lane, float (&facc)[NT][4]) {
    const int g = lane >> 2, t = lane & 3;
    const uint4 sg4 = reinterpret_cast<const uint4*>(sp + 3072)[g], sh4 = reinterpret_cast<const uint4*>(sp + 3072)[g + 8];
    const uint32_t sg[4] = {sg4.x ^ 0x80808080u, sg4.y ^ 0x80808080u, sg4.z ^ 0x80808080u, sg4.w ^ 0x80808080u};
    const uint32_t sh[4] = {sh4.x ^ 0x80808080u, sh4.y ^ 0x80808080u, sh4.z ^ 0x80808080u, sh4.w ^ 0x80808080u};
    const float dg = __half2float(reinterpret_cast<const __half*>(sp + 3328)[g]), dh = __half2float(reinterpret_cast<const __half*>(sp + 3328)[g + 8]);
    const uint4* xf = reinterpret_cast<const uint4*>(xc) + lane;
    float acc[NT == 1 ? 2 : NT][4];
#pragma unroll
    for (int n = 0; n < (NT == 1 ? 2 : NT); n++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[n][i] = 0.f;
#pragma unroll
    for (int half = 0; half < 2; half++) {
        uint32_t W[12];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const uint4 v = reinterpret_cast<const uint4*>(sp)[(3 * half + c) * 32 + lane];
            W[4 * c] = v.x; W[4 * c + 1] = v.y; W[4 * c + 2] = v.z; W[4 * c + 3] = v.w;
        }
#pragma unroll
        for (int G2 = 0; G2 < 4; G2++) {
            const uint32_t w0 = W[3 * G2], w1 = W[3 * G2 + 1], w2 = W[3 * G2 + 2];
            const uint32_t w3 = ((w0 << 6) & 0xc0c0c0c0u) | ((w1 << 4) & 0x30303030u) | ((w2 << 2) & 0x0c0c0c0cu);
            // bytes 4 (q - 32) + 128 under 1024: times scale / 4, less 288 scales
            const uint32_t r0 = (w0 & 0xfcfcfcfcu) ^ 0x80808080u, r1 = (w1 & 0xfcfcfcfcu) ^ 0x80808080u, r2 = (w2 & 0xfcfcfcfcu) ^ 0x80808080u, r3 = w3 ^ 0x80808080u;
            uint32_t a[2][4];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int j = 8 * half + 2 * G2 + h;
                const uint32_t s0 = h2_add(byte_h2(sg[j >> 2], j & 3), H_M1152), s1 = h2_add(byte_h2(sh[j >> 2], j & 3), H_M1152);
                const uint32_t m0 = h2_mul(s0, H_QUARTER), m1 = h2_mul(s1, H_QUARTER), c0 = h2_mul(s0, H_M288), c1 = h2_mul(s1, H_M288);
                const uint32_t x0 = h ? r2 : r0, x1 = h ? r3 : r1;
                a[h][0] = h2_fma(__byte_perm(x0, H_1024, 0x5250), m0, c0);
                a[h][1] = h2_fma(__byte_perm(x1, H_1024, 0x5250), m1, c1);
                a[h][2] = h2_fma(__byte_perm(x0, H_1024, 0x5351), m0, c0);
                a[h][3] = h2_fma(__byte_perm(x1, H_1024, 0x5351), m1, c1);
            }
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const uint4 bv = xf[n * (SG_FRAG / 16) + (4 * half + G2) * 32];
                mma16(acc[n], a[0][0], a[0][1], a[0][2], a[0][3], bv.x, bv.y);
                mma16(acc[NT == 1 ? 1 : n], a[1][0], a[1][1], a[1][2], a[1][3], bv.z, bv.w);
            }
        }
    }
    const float2* xd = reinterpret_cast<const float2*>(xc + NT * (SG_FRAG + SG_SUMS)) + t;
#pragma unroll
    for (int n = 0; n < NT; n++) {
        const float2 d = xd[n * 4];
        if (NT == 1) {
#pragma unroll
            for (int i = 0; i < 4; i++) acc[0][i] += acc[1][i];
        }
        facc[n][0] += d.x * dg * acc[n][0];
        facc[n][1] += d.y * dg * acc[n][1];
        facc[n][2] += d.x * dh * acc[n][2];
        facc[n][3] += d.y * dh * acc[n][3];
    }
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

template <int NT>
__global__ void __launch_bounds__(SG_THREADS, 1) gemm_sk_kernel(const __grid_constant__ SgArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[4], empty[4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kts = a.k >> 8, total = (a.tiles + SG_WARPS - 1) / SG_WARPS * kts;
    const int lo = share(blockIdx.x, total, gridDim.x), hi = share(blockIdx.x + 1, total, gridDim.x);
    constexpr int CHUNK = NT * SG_CHUNK;
    const int XS = a.x_slots;
    uint8_t* xring = smem;
    if (threadIdx.x == 0) {
        for (int s = 0; s < 4; s++) {
            bar_init(&full[s], 1);
            bar_init(&empty[s], SG_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_launch();
    if (warp == SG_WARPS) {
        pdl_wait();
        if (lane == 0) {
            int s = 0, kb = lo % kts;
            uint32_t turn = 0;
            for (int it = lo; it < hi; it++) {
                if (turn > 0 && !bar_wait(&empty[s], (turn - 1) & 1)) {
                    *(volatile int*)a.status = KS_TIMEOUT;
                    break;
                }
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&full[s])), "r"(CHUNK) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(smem_addr(xring + s * CHUNK)), "l"(a.x + (size_t)kb * CHUNK), "r"(CHUNK), "r"(smem_addr(&full[s])) : "memory");
                if (++kb == kts) kb = 0;
                if (++s == XS) {
                    s = 0;
                    turn++;
                }
            }
        }
        return;
    }
    // this warp's units, requested R - 1 items ahead
    const int R = a.ring;
    uint8_t* ring = smem + XS * CHUNK + (size_t)warp * R * a.slot_bytes;
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    int in_it = lo, in_slot = 0, in_kb = lo % kts, in_tile = lo / kts * SG_WARPS + warp;
    const uint8_t* in_p = nullptr;
    bool in_new = true, in_q6 = false;
    const uint32_t ring_lane = smem_addr(ring) + lane * 16;
    auto request = [&]() {
        if (in_it < hi) {
            if (in_new) {
                in_p = nullptr;
                if (in_tile < a.tiles) {
                    const TileAt ta = tile_at(a, in_tile, kts);
                    in_q6 = ta.ub == SG_UNIT_Q6K;
                    in_p = ta.p + (size_t)in_kb * ta.ub + lane * 16;
                }
                in_new = false;
            }
            if (in_p) {
                const uint32_t dst = ring_lane + in_slot * a.slot_bytes;
#pragma unroll
                for (int i = 0; i < 4; i++) cp16(dst + i * 512, in_p + i * 512, policy);
                if (in_q6) {
#pragma unroll
                    for (int i = 4; i < 6; i++) cp16(dst + i * 512, in_p + i * 512, policy);
                    if (lane < (SG_UNIT_Q6K - 3072) / 16) cp16(dst + 3072, in_p + 3072, policy);
                    in_p += SG_UNIT_Q6K;
                } else {
                    if (lane < (SG_UNIT_Q4K - 2048) / 16) cp16(dst + 2048, in_p + 2048, policy);
                    in_p += SG_UNIT_Q4K;
                }
            }
            if (++in_kb == kts) {
                in_kb = 0;
                in_new = true;
                in_tile += SG_WARPS;
            }
            in_it++;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        in_slot = in_slot + 1 == R ? 0 : in_slot + 1;
    };
    for (int i = 0; i < R - 1; i++) request();
    pdl_wait();

    const int g = lane >> 2, t = lane & 3;
    bool dead = false;
    int slot = 0, it = lo, xs = 0;
    uint32_t turn = 0;
    while (it < hi) {
        const int group = it / kts, kb0 = it - group * kts, seg_end = min(hi, (group + 1) * kts);
        const int tile = group * SG_WARPS + warp;
        const bool mine = tile < a.tiles;
        const TileAt ta = tile_at(a, mine ? tile : 0, kts);
        const bool q6 = ta.ub == SG_UNIT_Q6K;
        float facc[NT][4];
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) facc[n][i] = 0.f;
        const int n_seg = seg_end - it;
        for (; it < seg_end; it++) {
            request();
            if (R == 4) asm volatile("cp.async.wait_group 3;" ::: "memory");
            else if (R == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
            else asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            if (!dead && !__all_sync(0xffffffffu, bar_wait(&full[xs], turn & 1))) {
                dead = true;
                if (lane == 0) *(volatile int*)a.status = KS_TIMEOUT;
            }
            if (mine && !dead) {
                const uint8_t* sp = ring + slot * a.slot_bytes;
                const uint8_t* xc = xring + xs * CHUNK;
                if (q6) unit16_q6k<NT>(sp, xc, lane, facc);
                else unit16_q4k<NT>(sp, xc, lane, facc);
            }
            slot = slot + 1 == R ? 0 : slot + 1;
            __syncwarp();      // every lane is done with the unit and the chunk
            if (lane == 0) bar_arrive(&empty[xs]);
            if (++xs == XS) {
                xs = 0;
                turn++;
            }
        }
        if (!mine) continue;
        const int me = blockIdx.x * SG_WARPS + warp;
        if (kb0 != 0) {      // the group began in an earlier CTA: hand over the sums
            float* w = a.ws + (size_t)me * SG_WS_FLOATS;
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) w[(n * 4 + i) * 32 + lane] = facc[n][i];
            __threadfence();
            __syncwarp();
            if (lane == 0) st_release(&a.flags[me], 1u);
            continue;
        }
        // lane (g, t) holds rows g (i < 2) and g + 8 of x rows 8 n + 2 t + (i & 1).  What the results are added to is fetched ahead of the waits below, all of it at
        // once: loads that take turns with the stores cost 8 us of 24 at 32 rows.
        const float* bias = a.seg[0].bias;
        int out_off = a.seg[0].out_off;
#pragma unroll
        for (int i = 1; i < 4; i++)
            if (i == ta.s) {
                bias = a.seg[i].bias;
                out_off = a.seg[i].out_off;
            }
        const int row0 = ta.local * 16 + g;
        const float bias0 = bias ? bias[row0] : 0.f, bias1 = bias ? bias[row0 + 8] : 0.f;
        float* o = a.out + (a.mode == 2 ? (out_off + row0) >> 1 : out_off + row0);
        float old[NT][4];
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int b = 8 * n + 2 * t + (i & 1);
                old[n][i] = a.mode == 1 && b < a.nb ? __ldcg(o + (size_t)b * a.ldo + 8 * (i >> 1)) : 0.f;
            }
        if (n_seg < kts) {
            // the CTAs behind this one that hold the rest of the group: lane i watches the flag of the i-th (all at once: one after the other they cost a trip
            // to L2 each, 12 us of 16 for a product with nine parts a group)
            const int group_end = (group + 1) * kts;
            for (int c0 = blockIdx.x + 1; c0 < gridDim.x; c0 += 32) {
                const bool part = c0 + lane < gridDim.x && share(c0 + lane, total, gridDim.x) < group_end;
                const int n_parts = __popc(__ballot_sync(0xffffffffu, part));
                if (n_parts == 0) break;
                const int from = (c0 + lane) * SG_WARPS + warp;
                bool ok = true;
                if (part && !dead) {
                    ok = ld_acquire(&a.flags[from]) != 0u;
                    if (!ok) {
                        const unsigned long long t0 = now_ns();
                        while (!ok && now_ns() - t0 < SG_WAIT_NS) ok = ld_acquire(&a.flags[from]) != 0u;
                    }
                    if (!ok) *(volatile int*)a.status = KS_TIMEOUT;
                }
                if (!__all_sync(0xffffffffu, ok)) dead = true;
                const float* w = a.ws + ((size_t)c0 * SG_WARPS + warp) * SG_WS_FLOATS + lane;
#pragma unroll 4
                for (int c = 0; c < n_parts; c++)
#pragma unroll
                    for (int n = 0; n < NT; n++)
#pragma unroll
                        for (int i = 0; i < 4; i++) facc[n][i] += __ldcg(w + (size_t)c * SG_WARPS * SG_WS_FLOATS + (n * 4 + i) * 32);
                __syncwarp();
                if (part) a.flags[from] = 0u;
            }
        }
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int b = 8 * n + 2 * t + (i & 1);
                const float v = facc[n][i] + (i < 2 ? bias0 : bias1);
                float* at = o + (size_t)b * a.ldo;
                if (a.mode == 2) {      // the up value of a gate is one row further: lane + 4
                    const float up = __shfl_down_sync(0xffffffffu, v, 4);
                    if (!(g & 1) && b < a.nb) at[4 * (i >> 1)] = glu_act(v, up, a.act, a.alpha, a.limit);
                } else if (b < a.nb) {
                    at[8 * (i >> 1)] = v + old[n][i];
                }
            }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (dead)      // the producer may have chunks in flight: they land before the CTA leaves
        for (int i = max(0, hi - lo - XS); i < hi - lo; i++) bar_wait(&full[i % XS], (i / XS) & 1);
}

// One warp per (row, 256-block): eight columns per lane.  A row that is normalised belongs to one CTA (its sum of squares is needed first).
// Rows nb .. 8 ceil(nb / 8) - 1 of the last group are written as zeros.
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

__device__ __forceinline__ void store_block(const Rows16Args& a, int nt, int ntile, int gg, int blk, int lane, const float (&v)[8]) {
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) m = fmaxf(m, fabsf(v[i]));
    m = warp_max(m);
    const int e = max((int)(__float_as_uint(m) >> 23), 16);                        // scale 2^(e - 135): the largest value lands in 256..512
    const float inv = __uint_as_float((uint32_t)(262 - e) << 23), scale = __uint_as_float((uint32_t)(e - 8) << 23);
    __half h[8];
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        h[i] = __float2half_rn(v[i] * inv);
        sum += __half2float(h[i]);
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);                                    // the 32 columns of four lanes
    uint8_t* c = a.out + (size_t)blk * nt * SG_CHUNK;
    // lane: columns 8 lane .. + 7 of the block = t values 2 (lane & 1) and + 1 of 16-column group lane / 2, fragment pair lane / 4
    __half2* f = reinterpret_cast<__half2*>(c + ntile * SG_FRAG + ((size_t)(lane >> 2) * 32 + gg * 4 + 2 * (lane & 1)) * 16 + ((lane >> 1) & 1) * 8);
    f[0] = __halves2half2(h[0], h[2]);
    f[1] = __halves2half2(h[1], h[3]);
    f[4] = __halves2half2(h[4], h[6]);
    f[5] = __halves2half2(h[5], h[7]);
    // sums of sub-blocks 2t, 2t + 1: lanes 8 t and 8 t + 4 hold them
    const float next = __shfl_down_sync(0xffffffffu, sum, 4);
    if ((lane & 7) == 0) {
        const __half h0 = __float2half_rn(sum), h1 = __float2half_rn(next);
        __half2* s = reinterpret_cast<__half2*>(c + nt * SG_FRAG + ntile * SG_SUMS + (gg * 4 + (lane >> 3)) * 8);
        s[0] = __halves2half2(h0, h1);
        s[1] = __halves2half2(__float2half_rn(sum - __half2float(h0)), __float2half_rn(next - __half2float(h1)));
    }
    if (lane == 0) *reinterpret_cast<float*>(c + nt * (SG_FRAG + SG_SUMS) + (ntile * 8 + gg) * 4) = scale;
}

template <bool BF16>
__global__ void __launch_bounds__(R16_WARPS * 32) rows16_kernel(const __grid_constant__ Rows16Args a, int nb) {
    __shared__ float ssq[R16_WARPS];
    pdl_launch();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = blockIdx.x, nkb = a.k >> 8, nt = gridDim.x >> 3;
    const int ntile = row >> 3, gg = row & 7;
    const int b0 = blockIdx.y * R16_WARPS + warp, step = gridDim.y * R16_WARPS;
    const bool pad = row >= nb;
    if (!a.norm_w) {
        for (int blk = b0; blk < nkb; blk += step) {
            float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (!pad) load8<BF16>(a.x, (size_t)row * a.ldx + blk * 256 + lane * 8, v);
            store_block(a, nt, ntile, gg, blk, lane, v);
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
        store_block(a, nt, ntile, gg, blk, lane, v[i]);
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
B2_API long long b2_rows16_bytes(int nb, int k) { return (long long)(k >> 8) * ((nb + 7) >> 3) * SG_CHUNK; }

// Rows in the order that b2_gemm_sk reads.  k a multiple of 256 (at most 16384 with a norm), x and out 16-byte aligned, ldx a multiple of 8 (fp32: of 4).
B2_API int b2_rows16(const Rows16Args* in, int nb, int pdl, cudaStream_t st) {
    Rows16Args a = *in;
    if (nb < 1 || nb > 32 || a.k < 256 || (a.k & 255) || !a.x || !a.out || (((uintptr_t)a.x | (uintptr_t)a.out | (uintptr_t)a.norm_w) & 15) || (a.ldx & (a.bf16 ? 7 : 3)))
        return (int)cudaErrorInvalidValue;
    if (a.norm_w && (a.k >> 8) > R16_WARPS * R16_KEEP) return (int)cudaErrorNotSupported;
    const int nkb = a.k >> 8, rows = (nb + 7) & ~7;
    void* args[] = {&a, &nb};
    const dim3 grid(rows, a.norm_w ? 1 : (nkb + R16_WARPS - 1) / R16_WARPS);
    return go(a.bf16 ? (const void*)rows16_kernel<true> : (const void*)rows16_kernel<false>, grid, dim3(R16_WARPS * 32), 0, args, st, pdl);
}

// y = W x for 1..32 rows in the chunks of b2_rows16, up to four matrices of one row length.  Returns a cudaError_t value.
B2_API int b2_gemm_sk(const SgArgs* in, int max_ctas, int pdl, cudaStream_t st) {
    SgArgs a = *in;
    if (a.nseg < 1 || a.nseg > 4 || a.nb < 1 || a.nb > 32 || a.k < 256 || (a.k & 255) || !a.x || ((uintptr_t)a.x & 15) || !a.out || !a.ws || !a.flags || !a.status || a.mode < 0 ||
        a.mode > 2)
        return (int)cudaErrorInvalidValue;
    int slot = 0, tiles = 0;
    for (int s = 0; s < a.nseg; s++) {
        SgSeg& g = a.seg[s];
        if ((g.type != WT_Q4_K && g.type != WT_Q6_K) || g.n <= 0 || (g.n & 15) || ((uintptr_t)g.w & 15) || (a.mode == 2 && (g.out_off & 1))) return (int)cudaErrorInvalidValue;
        g.tile0 = tiles;
        tiles += g.n >> 4;
        slot = slot > (g.type == WT_Q6_K ? SG_UNIT_Q6K : SG_UNIT_Q4K) ? slot : (g.type == WT_Q6_K ? SG_UNIT_Q6K : SG_UNIT_Q4K);
    }
    const int nt = a.nb <= 8 ? 1 : a.nb <= 16 ? 2 : a.nb <= 24 ? 3 : 4;
    a.tiles = tiles;
    a.slot_bytes = slot;
    const size_t chunk = (size_t)nt * SG_CHUNK;
    // weights in flight first: four slots a warp where they fit beside three chunks
    a.ring = SG_WARPS * 4 * slot + 3 * chunk <= SG_MAX_SMEM ? 4 : 3;
    a.x_slots = (SG_MAX_SMEM - (size_t)SG_WARPS * a.ring * slot) / chunk >= 4 ? 4 : 3;
    const size_t smem = SG_WARPS * a.ring * slot + a.x_slots * chunk;
    if (smem > SG_MAX_SMEM) return (int)cudaErrorInvalidValue;
    const void* fn = nt == 1 ? (const void*)gemm_sk_kernel<1> : nt == 2 ? (const void*)gemm_sk_kernel<2> : nt == 3 ? (const void*)gemm_sk_kernel<3> : (const void*)gemm_sk_kernel<4>;
    static PerDeviceOnce once[4];
    if (once[nt - 1].first()) {
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SG_MAX_SMEM);
        if (e != cudaSuccess) return (int)e;
    }
    const int total = (tiles + SG_WARPS - 1) / SG_WARPS * (a.k >> 8);
    if (total >= 1 << 23) return (int)cudaErrorNotSupported;
    int grid = total < sms() ? total : sms();      // one CTA per SM: all are resident, so waits on other CTAs end
    if (grid > 4096 / SG_WARPS) grid = 4096 / SG_WARPS;
    if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
    void* args[] = {&a};
    return go(fn, dim3((unsigned)grid), dim3(SG_THREADS), smem, args, st, pdl);
}
