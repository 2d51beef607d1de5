// Mixture-of-experts products on MXFP4 experts for decode steps and prompts, sm_100a: every (token, expert) pair's row times the expert's matrix, each expert's
// blocks read once for all rows that chose it, up to 64 at a time.
//
// The bound is the stream of 4-bit blocks (13 MB an expert of gpt-oss-120b).  What the earlier forms cost on top of it: one grid row per pair read an expert again
// for each of its tokens and spent dp4a on every copy (280 us a layer at 16 tokens, 194 here, stream 105); a tcgen05 form with tokens as its 128 rows padded every expert
// to 128 of them and expanded the codes to bf16 (1341 us at 1024 tokens, 769 here, stream 258).
// Expanding codes in registers for mma.sync was no way out: its integer instructions alone took 1000 cycles per 32 x 128 codes of a warp (1535 us at 1024 tokens).  Here nothing
// is expanded:
//   * tcgen05.mma kind::mxf8f6f4 multiplies E2M1 codes under their own E8M0 block scales: 128 matrix rows are the M of a tile, the rows of the pairs its N.  The codes only
//     move to the 8-bytes-in-16 form that the instruction reads (two 8-byte stores a 32-column block), the scales go to tensor memory with tcgen05.cp.
//   * A row is rounded to bf16 and split into two E4M3 values with block scales of their own: eight significant bits are four and four, so that the two add up to the bf16 value
//     (to 2^-18 of the block's largest value).  They are two rows of N; the epilogue adds their columns.
//   * The codes of a 32-column block are stored as bytes of columns c and 16 + c; the rows are written in that order of columns too (moe_rows_kernel), tile by tile in the layout
//     and swizzle that shared memory has, so that a step's rows are one bulk copy; the scales of a tile's matrix rows are one more.
//   * What bounds it now is the path through L1 and shared memory: 660 cycles a step of 128 x 128 codes at eight rows, in which a product of 32 columns takes 70 cycles to fetch its
//     128 matrix rows however few rows it has (280 a step) and the loads and stores of the codes 256.  Three CTAs an SM with two stages each are best up to 24 rows (two with three
//     stages 10 % slower; four leave the L1 too small for the loads under way, 70 % slower), two from 32 rows on.  128 bytes of a matrix row per request instead of 64 cost 10 %
//     (the stores fall apart), 16-byte stores with the padding 10 %; codes through a cp.async ring in shared memory instead of registers, and two teams of warps that bring
//     alternate steps, 20 % at eight rows (two CTAs fit) and nothing at 48.
#include <cuda_fp8.h>

#include "tc_common.cuh"

using namespace tc;

__device__ int g_moe_status = 0;

namespace {

constexpr int STEP = 128;                           // columns per step: four blocks, one of each for the four products of 32 columns
constexpr int STAGES = 2, AHEAD = 4;                // steps in shared memory, steps whose codes are under way to registers
constexpr int MAX_SMEM = 225 * 1024, MAX_K = 16384;
constexpr int A_BYTES = 128 * STEP, SF_BYTES = 512; // a step's codes (a byte each in shared memory), its scales of up to 128 rows

__host__ __device__ constexpr int x_step_bytes(int rows) { return 2 * rows * STEP + SF_BYTES; }      // both parts of the chunk's rows and their scales

// Scales in the order that tcgen05.cp 32x128b takes: row r, block b of a step.
__host__ __device__ constexpr int sf_at(int r, int b) { return (r & 31) * 16 + (r >> 5) * 4 + b; }

}  // namespace

struct MoeSortArgs {
    const int* lids;       // [pairs] expert on this GPU, or -1
    int pairs, n_experts;  // n_experts <= 512
    int rows;              // rows per chunk, a multiple of 8
    int max_chunks;
    int* chunks;           // [1 + 2 max_chunks]: number of chunks, then (expert, rows) of each
    int* row_of_pair;      // [pairs] chunk * rows + place, or -1
    int* pair_of_row;      // [max_chunks * rows]
};

// One CTA: count, scan, hand out rows.  The order of the pairs inside an expert depends on the atomics, the value computed for a pair does not.
__global__ void __launch_bounds__(1024) moe_sort_kernel(const __grid_constant__ MoeSortArgs a) {
    __shared__ int cnt[512], first[512], cur[512], sums[16];
    pdl_launch();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int e = tid; e < 512; e += 1024) cnt[e] = cur[e] = 0;
    __syncthreads();
    for (int p = tid; p < a.pairs; p += 1024) {
        const int l = a.lids[p];
        if (l >= 0 && l < a.n_experts) atomicAdd(&cnt[l], 1);
    }
    __syncthreads();
    int mine = 0, scan = 0;
    if (tid < 512) {       // chunks of this expert, and of those before it
        mine = (cnt[tid] + a.rows - 1) / a.rows;
        scan = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, scan, o);
            if (lane >= o) scan += v;
        }
        if (lane == 31) sums[warp] = scan;
    }
    __syncthreads();
    if (tid < 512) {
        int before = scan - mine;
        for (int w = 0; w < warp; w++) before += sums[w];
        first[tid] = before;
        for (int c = 0; c < mine; c++)
            if (before + c < a.max_chunks) {
                a.chunks[1 + 2 * (before + c)] = tid;
                a.chunks[2 + 2 * (before + c)] = min(a.rows, cnt[tid] - c * a.rows);
            }
        if (tid == 511) a.chunks[0] = min(before + mine, a.max_chunks);
    }
    __syncthreads();
    for (int p = tid; p < a.pairs; p += 1024) {
        const int l = a.lids[p];
        int r = -1;
        if (l >= 0 && l < a.n_experts) r = first[l] * a.rows + atomicAdd(&cur[l], 1);
        if (r >= a.max_chunks * a.rows) r = -1;
        a.row_of_pair[p] = r;
        if (r >= 0) a.pair_of_row[r] = p;
    }
}

// Row p / per_token of x (fp32 or bf16) to the pair's place in the chunks of `rows` rows; without row_of_pair, row p of x to place p where a chunk has such a row.  Two threads per
// 32-column block: one has columns 0-7 and 16-23, the other the rest, which are 16 bytes of the result each (a lane per column, a byte per store: 35 us for 4096 rows of 2880).
// The columns that fill the last step are zeros.
template <bool BF16>
__global__ void __launch_bounds__(256) moe_rows_kernel(const void* x, int ldx, int cols, int per_token, const int* row_of_pair, const int* chunks, int rows, uint8_t* out) {
    pdl_launch();
    pdl_wait();
    const int p = blockIdx.x, steps = (cols + STEP - 1) / STEP;
    int r = p;
    if (row_of_pair) {
        r = row_of_pair[p];
        if (r < 0) return;
    } else if (p / rows >= chunks[0] || p % rows >= chunks[2 + 2 * (p / rows)]) {
        return;
    }
    const int place = r % rows;
    const size_t at = (size_t)(row_of_pair ? p / per_token : p) * ldx;
    uint8_t* to = out + (size_t)(r / rows) * steps * x_step_bytes(rows);
    for (int i0 = 0; i0 < 8 * steps; i0 += 256) {
        const int i = i0 + threadIdx.x, b = i >> 1, c = 32 * b + 8 * (i & 1);
        float v[16];      // columns c .. c + 7, c + 16 .. c + 23, rounded to bf16
        if (c >= cols) {
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = 0.f;
        } else {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (BF16) {
                    const uint4 w = *reinterpret_cast<const uint4*>((const __nv_bfloat16*)x + at + c + 16 * h);
                    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int j = 0; j < 8; j++) v[8 * h + j] = __uint_as_float(j & 1 ? u[j >> 1] & 0xFFFF0000u : u[j >> 1] << 16);
                } else {
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const float4 w = *reinterpret_cast<const float4*>((const float*)x + at + c + 16 * h + 4 * q);
                        const float u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int j = 0; j < 4; j++) v[8 * h + 4 * q + j] = __bfloat162float(__float2bfloat16_rn(u[j]));
                    }
                }
            }
        }
        uint32_t bad = 0;      // no finite numbers: NaN
#pragma unroll
        for (int j = 0; j < 16; j++) bad |= (uint32_t)!(fabsf(v[j]) <= 3.4e38f) << j;
        uint8_t* tile = to + (size_t)(b >> 2) * x_step_bytes(rows);
        const int chunk16 = 2 * (b & 3) + (i & 1);
#pragma unroll
        for (int part = 0; part < 2; part++) {
            float m = 0.f;
#pragma unroll
            for (int j = 0; j < 16; j++) m = fmaxf(m, bad >> j & 1 ? 0.f : fabsf(v[j]));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            // the block's largest value in [128, 256) of the scale
            const int eb = max((int)(__float_as_uint(m) >> 23) - 7, 1);
            const float down = __uint_as_float((uint32_t)(254 - eb) << 23), up = __uint_as_float((uint32_t)eb << 23);
            uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int j = 0; j < 8; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {      // byte 2 j + h: column c + j + 16 h
                    const int e = 8 * h + j;
                    const __nv_fp8_storage_t q = bad >> e & 1 ? 0x7F : __nv_cvt_float_to_fp8(v[e] * down, __NV_SATFINITE, __NV_E4M3);
                    v[e] -= __half2float(__half(__nv_cvt_fp8_to_halfraw(q, __NV_E4M3))) * up;
                    w[j >> 1] |= (uint32_t)q << (16 * (j & 1) + 8 * h);
                }
            if (i >= 8 * steps) continue;
            const int n = part * rows + place;
            *reinterpret_cast<uint4*>(tile + n * STEP + ((chunk16 ^ (n & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
            if (!(i & 1)) tile[2 * rows * STEP + sf_at(n, b & 3)] = (uint8_t)eb;
        }
    }
}

struct MoeFp4Args {
    const uint8_t* q;         // [experts * n][k / 2] codes: low nibbles of a 32-block's 16 bytes are its first 16 columns
    const uint8_t* s;         // [experts * n][k / 32] E8M0
    const float* bias;        // [experts * n] or null
    int n, k;                 // n a multiple of 16, k of 32
    const uint8_t* x;         // the rows as moe_rows_kernel writes them
    const int* chunks;
    const int* pair_of_row;   // or null: results stay at the rows' places
    void* out;                // glu: bf16 [chunk rows][n / 2]; else fp32 [pairs][n], or [chunk rows][n] without pair_of_row
    int glu;                  // 0: off, 1 + activation otherwise (matrix rows 2i / 2i + 1 = gate / up of output i)
    float alpha, limit;
};

namespace {

// E2M1 x E4M3 under E8M0 scales of 32 columns -> fp32, 128 x n, both K-major; `block` picks the byte of the scales' words.
__device__ __forceinline__ constexpr uint32_t mx_idesc(int n, int block) {
    return ((uint32_t)block << 4) | (5u << 7) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | (1u << 27) | ((uint32_t)block << 29);
}
__device__ __forceinline__ void umma_mx(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], %1, %2, %3, [%4], [%5], p;\n\t}"
                 ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate) : "memory");
}
// 512 bytes of scales (32 rows of 16 bytes, 8-row groups 128 bytes apart, no swizzle) to four columns of tensor memory.
__device__ __forceinline__ void scales_to_tmem(uint32_t taddr, const void* src) {
    const uint64_t desc = (uint64_t)((smem_u32(src) & 0x3FFFF) >> 4) | (uint64_t)(128 >> 4) << 32 | (uint64_t)1 << 46;
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}
// Eight columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr));
}

// One CTA = 128 matrix rows x a chunk of R rows.  Warps 0 to 3 bring the codes and do the epilogue, warp 4 asks for the rows, warp 5 multiplies.
template <int R>
__global__ void __launch_bounds__(192, 3) moe_fp4_kernel(const __grid_constant__ MoeFp4Args a) {
    constexpr int N = 2 * R, XB = x_step_bytes(R), X_STAGE = XB + SF_BYTES;      // tiles start at multiples of 1024 bytes
    constexpr int COLS = N + 8 * STAGES <= 64 ? 64 : N + 8 * STAGES <= 128 ? 128 : 256;      // accumulators, then eight columns of scales per stage
    extern __shared__ __align__(1024) uint8_t raw[];
    uint8_t* sm = (uint8_t*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    uint8_t* codes = sm;
    uint8_t* xs = sm + STAGES * A_BYTES;
    uint8_t* sfa = xs + STAGES * X_STAGE;
    uint8_t* scales = sfa + STAGES * SF_BYTES;      // [128][k / 32] of the tile's rows, which are contiguous in memory
    __shared__ uint64_t full_a[STAGES], full_x[STAGES], empty[STAGES], full_s, done;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_failed;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_failed = 0;
        for (int s = 0; s < STAGES; s++) {
            mbar_init(&full_a[s], 128);
            mbar_init(&full_x[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&full_s, 1);
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch();      // not before the tensor memory is there: CTAs of the next kernel that came first would keep it until this one ends
    pdl_wait();
    const uint32_t tmem = tmem_slot;
    const int chunk = blockIdx.y, steps = (a.k + STEP - 1) / STEP, blocks = a.k >> 5, row0 = blockIdx.x * 128;
    if (chunk < a.chunks[0]) {
        const int e = a.chunks[1 + 2 * chunk], count = a.chunks[2 + 2 * chunk];
        if (warp < 4) {
            // block t of rows row0 + 32 j + i in every step; rows beyond the matrix repeat its last one (their results are not stored)
            const int t = tid & 3, i = tid >> 2;
            const uint8_t* qp[4];
#pragma unroll
            for (int j = 0; j < 4; j++) qp[j] = a.q + ((size_t)e * a.n + min(row0 + 32 * j + i, a.n - 1)) * (size_t)(a.k >> 1) + 16 * t;
            uint4 q[AHEAD][4];
            auto fetch = [&](int st, uint4 (&qs)[4]) {
                const bool in = 4 * st + t < blocks;
#pragma unroll
                for (int j = 0; j < 4; j++) qs[j] = in ? ldg16(qp[j] + 64 * st) : make_uint4(0u, 0u, 0u, 0u);
            };
#pragma unroll
            for (int d = 0; d < AHEAD; d++)
                if (d < steps) fetch(d, q[d]);
            bool ok = mbar_wait(&full_s, 0);
            for (int st0 = 0; st0 < steps && ok; st0 += AHEAD) {
#pragma unroll
                for (int d = 0; d < AHEAD; d++) {
                    const int st = st0 + d;
                    if (st >= steps || !ok) break;
                    const int stage = st % STAGES;
                    if (st >= STAGES) ok = mbar_wait(&empty[stage], (st / STAGES - 1) & 1);
                    if (!ok) break;
                    uint8_t* to = codes + stage * A_BYTES;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const int r = 32 * j + i;      // r & 7 = i & 7
                        *reinterpret_cast<uint2*>(to + r * STEP + (((2 * t) ^ (r & 7)) << 4)) = make_uint2(q[d][j].x, q[d][j].y);
                        *reinterpret_cast<uint2*>(to + r * STEP + (((2 * t + 1) ^ (r & 7)) << 4)) = make_uint2(q[d][j].z, q[d][j].w);
                    }
                    uint32_t sc = 0x7F7F7F7Fu;      // of row tid; no NaN behind the row's end
                    const uint8_t* at = scales + tid * blocks + 4 * st;
                    if (!(blocks & 1)) {
                        if (4 * st + 2 <= blocks) sc = (sc & 0xFFFF0000u) | *reinterpret_cast<const uint16_t*>(at);
                        if (4 * st + 4 <= blocks) sc = (sc & 0x0000FFFFu) | (uint32_t)*reinterpret_cast<const uint16_t*>(at + 2) << 16;
                    } else {
#pragma unroll
                        for (int h = 0; h < 4; h++)
                            if (4 * st + h < blocks) sc = (sc & ~(0xFFu << (8 * h))) | (uint32_t)at[h] << (8 * h);
                    }
                    *reinterpret_cast<uint32_t*>(sfa + stage * SF_BYTES + sf_at(tid, 0)) = sc;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full_a[stage])) : "memory");
                    if (st + AHEAD < steps) fetch(st + AHEAD, q[d]);
                }
            }
            ok = ok && mbar_wait(&done, 0);
            if (!ok) s_failed = 1;
            tc_fence_after();
            const int row = row0 + 32 * warp + lane, x0 = chunk * R;
            const float bias = a.bias && row < a.n ? a.bias[(size_t)e * a.n + row] : 0.f;
            ok = __all_sync(0xffffffffu, ok);
#pragma unroll
            for (int n0 = 0; n0 < R; n0 += 8) {
                if (n0 >= count || !ok) break;
                uint32_t hi[8], lo[8];
                tmem_ld8(tmem + ((uint32_t)(32 * warp) << 16) + n0, hi);
                tmem_ld8(tmem + ((uint32_t)(32 * warp) << 16) + R + n0, lo);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float v = __uint_as_float(hi[j]) + __uint_as_float(lo[j]) + bias;
                    if (a.glu) {
                        const float up = __shfl_down_sync(0xffffffffu, v, 1);
                        if (!(lane & 1) && row < a.n && n0 + j < count)
                            ((__nv_bfloat16*)a.out)[(size_t)(x0 + n0 + j) * (a.n >> 1) + (row >> 1)] = __float2bfloat16_rn(glu_act(v, up, a.glu - 1, a.alpha, a.limit));
                    } else if (row < a.n && n0 + j < count) {
                        ((float*)a.out)[(size_t)(a.pair_of_row ? a.pair_of_row[x0 + n0 + j] : x0 + n0 + j) * a.n + row] = v;
                    }
                }
            }
            tc_fence_before();
        } else if (warp == 4) {
            if (lane == 0) {
                const uint8_t* src = a.x + (size_t)chunk * steps * XB;
                bool ok = true;
                const int bytes = min(128, a.n - row0) * blocks;
                mbar_expect_tx(&full_s, bytes);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(scales)),
                             "l"(a.s + ((size_t)e * a.n + row0) * blocks), "r"(bytes), "r"(smem_u32(&full_s)) : "memory");
                int st = 0;
                for (; st < steps; st++) {
                    const int stage = st % STAGES;
                    if (st >= STAGES) ok = mbar_wait(&empty[stage], (st / STAGES - 1) & 1);
                    if (!ok) break;
                    mbar_expect_tx(&full_x[stage], XB);
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(xs + stage * X_STAGE)),
                                 "l"(src + (size_t)st * XB), "r"(XB), "r"(smem_u32(&full_x[stage])) : "memory");
                }
                if (!ok) {      // copies under way land before the CTA leaves
                    s_failed = 1;
                    mbar_wait(&full_s, 0);
                    for (int i = st - STAGES; i < st; i++) mbar_wait(&full_x[i % STAGES], (i / STAGES) & 1);
                }
            }
        } else if (lane == 0) {
            bool ok = true;
            int st = 0;
            for (; st < steps; st++) {
                const int stage = st % STAGES, phase = (st / STAGES) & 1;
                ok = mbar_wait(&full_x[stage], phase) && mbar_wait(&full_a[stage], phase);
                if (!ok) break;
                tc_fence_after();
                const uint32_t ta = tmem + N + 8 * stage, tb = ta + 4;
                const uint8_t* x = xs + stage * X_STAGE;
                scales_to_tmem(ta, sfa + stage * SF_BYTES);
                scales_to_tmem(tb, x + N * STEP);
                const uint64_t adesc = umma_desc(codes + stage * A_BYTES), bdesc = umma_desc(x);
#pragma unroll
                for (int b = 0; b < 4; b++) umma_mx(tmem, adesc + 2 * b, bdesc + 2 * b, mx_idesc(N, b), ta, tb, st != 0 || b != 0);
                umma_commit(&empty[stage]);
            }
            if (ok) {
                umma_commit(&done);
            } else {      // products under way end, and copies that the other warp asked for, before the CTA leaves
                s_failed = 1;
                for (int i = max(0, st - STAGES); i < st; i++) mbar_wait(&empty[i % STAGES], (i / STAGES) & 1);
                for (int i = st; i < min(st + STAGES, steps); i++) mbar_wait(&full_x[i % STAGES], (i / STAGES) & 1);
            }
        }
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
    if (tid == 0 && s_failed) atomicExch(&g_moe_status, (int)KS_TIMEOUT);
}

int go(const void* fn, dim3 grid, dim3 block, void** args, cudaStream_t st, int pdl, int smem = 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelExC(&cfg, fn, args);
}

template <int R>
int launch(const MoeFp4Args& a, int max_chunks, int pdl, cudaStream_t st) {
    const int smem = 1024 + STAGES * (A_BYTES + x_step_bytes(R) + 2 * SF_BYTES) + 128 * (a.k >> 5);
    if (smem > MAX_SMEM) return (int)cudaErrorNotSupported;
    static PerDeviceOnce once;
    if (once.first()) cudaFuncSetAttribute(moe_fp4_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM);
    // No more shared memory than the CTAs need (1 KB each of static and of reserved memory): the rest is the L1 that the loads under way live in.  Left to itself the SM keeps the
    // split of a kernel before it: 16 tokens behind a GEMM of 200 KB took 173 us instead of 109.
    // At least 36 KB of it: with three CTAs of 32 to 48 rows an SM kept 3 to 27 KB, and 2048 pairs of 128 experts took 864 us at 32 rows, 677 with two CTAs.
    const int fit = 192 * 1024 / (smem + 2048), ctas = fit < 1 ? 1 : fit < 3 ? fit : 3;
    cudaFuncSetAttribute(moe_fp4_kernel<R>, cudaFuncAttributePreferredSharedMemoryCarveout, (ctas * (smem + 2048) * 100 + 228 * 1024 - 1) / (228 * 1024));
    MoeFp4Args copy = a;
    void* args[] = {&copy};
    return go((const void*)moe_fp4_kernel<R>, dim3((unsigned)((a.n + 127) / 128), (unsigned)max_chunks), dim3(192), args, st, pdl, smem);
}

}  // namespace

B2_API int b2_moe_sort(const MoeSortArgs* in, int pdl, cudaStream_t st) {
    MoeSortArgs a = *in;
    if (a.pairs < 1 || a.n_experts < 1 || a.n_experts > 512 || a.rows < 8 || (a.rows & 7) || a.max_chunks < 1) return (int)cudaErrorInvalidValue;
    void* args[] = {&a};
    return go((const void*)moe_sort_kernel, dim3(1), dim3(1024), args, st, pdl);
}

// Bytes of `chunks` chunks of `rows` rows of `cols` columns.
B2_API long long b2_moe_rows_bytes(int chunks, int rows, int cols) { return (long long)chunks * ((cols + STEP - 1) / STEP) * x_step_bytes(rows); }

// x: fp32 or bf16 rows of cols columns (a multiple of 32), ldx apart, 16-byte aligned.  row_of_pair null: `pairs` rows at their places (x has chunks * rows of them).
B2_API int b2_moe_rows(const void* x, int bf16, int ldx, int cols, int per_token, const int* row_of_pair, const int* chunks, int rows, int pairs, void* out, int pdl,
                       cudaStream_t st) {
    if (!x || !out || !chunks || pairs < 1 || per_token < 1 || cols < 32 || (cols & 31) || (ldx & (bf16 ? 7 : 3)) || rows < 8 || rows > 64 || (rows & 7) ||
        (((uintptr_t)x | (uintptr_t)out) & 15)) return (int)cudaErrorInvalidValue;
    uint8_t* o = (uint8_t*)out;
    void* args[] = {&x, &ldx, &cols, &per_token, &row_of_pair, &chunks, &rows, &o};
    return go(bf16 ? (const void*)moe_rows_kernel<true> : (const void*)moe_rows_kernel<false>, dim3(pairs), dim3(256), args, st, pdl);
}

// chunk_rows: 8, 16, 24, 32, 48 or 64, what moe_sort and moe_rows were given.  Returns a cudaError_t value (cudaErrorNotSupported: other shapes; nothing launched).
B2_API int b2_moe_fp4(const MoeFp4Args* in, int chunk_rows, int max_chunks, int pdl, cudaStream_t st) {
    const MoeFp4Args a = *in;
    if (!a.q || !a.s || !a.x || !a.chunks || !a.out || max_chunks < 1 || max_chunks > 65535 || a.glu < 0 || a.glu > 3 || (((uintptr_t)a.q | (uintptr_t)a.s | (uintptr_t)a.x) & 15))
        return (int)cudaErrorInvalidValue;
    if (a.n < 16 || (a.n & 15) || a.k < 32 || (a.k & 31) || a.k > MAX_K) return (int)cudaErrorNotSupported;
    switch (chunk_rows) {
        case 8: return launch<8>(a, max_chunks, pdl, st);
        case 16: return launch<16>(a, max_chunks, pdl, st);
        case 24: return launch<24>(a, max_chunks, pdl, st);
        case 32: return launch<32>(a, max_chunks, pdl, st);
        case 48: return launch<48>(a, max_chunks, pdl, st);
        case 64: return launch<64>(a, max_chunks, pdl, st);
    }
    return (int)cudaErrorInvalidValue;
}

// Nonzero if a wait ran out since the last call; resets it.
B2_API int b2_moe_fp4_status() {
    int v = 0, zero = 0;
    cudaMemcpyFromSymbol(&v, g_moe_status, sizeof(int));
    if (v) cudaMemcpyToSymbol(g_moe_status, &zero, sizeof(int));
    return v;
}
