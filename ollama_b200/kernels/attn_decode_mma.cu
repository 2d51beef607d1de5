// Split-K decode attention on the tensor cores, sm_100a.
//
// Same contract as the scalar kernel of attn_decode.cu (one query token per sequence, partial results
// (max, sum, unnormalised output) per split, merged by the combine kernel), different inner loop: the
// query heads that share a KV head are the rows of an m16n8k16 MMA tile (grouped-query attention gives
// 4..16 such heads; missing rows are zero), so one tile of 64 cached positions costs each warp 32 MMAs
// instead of some 1800 scalar instructions per 16 positions.  grid = (splits, kv heads, sequences), 4 warps.
// Cache rows arrive in shared memory through cp.async; every warp keeps its own running soft-max statistics and output accumulator, and the four warps are merged
// through shared memory at the end.  The scalar kernel stays the choice for short contexts and for head sizes without an instantiation here.
// Two kernels: of flat caches every warp streams turns of 16 positions of its own (below); the paged one reads tiles of 64 positions, a page, that the four warps share (16 each), starts at the
// query's chunk or window (keys that are kept in front of a window come first), and normalises q and k over their whole projections or heads before the rotation.
// Both take two stages of shared memory (int8 caches three), or three / four when the launch has so few CTAs that each SM holds two / one.
#include "attn_args.cuh"
#include "rows.cuh"

namespace {

constexpr int BN = 64, PAD = 8, ROWS = 16;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Four int8 values times a block's scale, as two f16 pairs, each rounded once (1024 + 128 + value under the exponent of 1024, less 1152, is exact).
__device__ __forceinline__ uint2 expand_q8x4(uint32_t w, __half2 d) {
    w ^= 0x80808080u;
    uint32_t lo = __byte_perm(w, 0x64646464u, 0x4140), hi = __byte_perm(w, 0x64646464u, 0x4342);
    const __half2 base = __half2half2(__ushort_as_half(0x6480));
    const __half2 a = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&lo), base), d), b = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&hi), base), d);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

template <int D, int NS>
__global__ void __launch_bounds__(128) attn_decode_paged_kernel(const __grid_constant__ AttnDecodeArgs a, const __grid_constant__ AttnRopeArgs r) {
    constexpr int LD = D + PAD, TS = NS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __half* sQ = reinterpret_cast<__half*>(smem_raw);            // [ROWS][LD]
    __half* sK = sQ + ROWS * LD;                                 // [TS][BN][LD]
    __half* sV = sK + TS * BN * LD;                              // [TS][BN][LD]
    __shared__ float s_m[4][ROWS], s_l[4][ROWS];
    __shared__ float s_cs[128], s_sn[128];                        // cos / sin of the query position per rotated pair (fused form)
    __shared__ __half s_newk[D], s_newv[D];                       // the query token's own key and value rows (fused form, owning split)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
    const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
    const int group = a.n_heads / a.n_kv_heads;                  // query heads per KV head (<= ROWS, checked by the launcher)
    const int head0 = kvh * group;

    pdl_launch();
    pdl_wait();
    const int qpos = a.positions[b], slot = a.slots[b];
    const int kv_len = qpos + 1;
    const int start = first_key(qpos, a.chunk, a.window);
    const int base = start & ~(BN - 1);                         // tiles begin at page borders
    // the keys to visit, numbered from 0: `front` of them at the sequence's start (whole tiles with kept keys), the rest `shift` positions further on
    const int front = a.window > 0 ? BN * kept_tiles(a.keep, base, BN) : 0, shift = base - front, keep = a.keep;
    const int span = kv_len - shift;
    int chunk = (span + a.n_splits - 1) / a.n_splits;
    chunk = ((chunk + BN - 1) / BN) * BN;
    const int p0 = split * chunk, p1 = min(p0 + chunk, span);
    const int n_tiles = p1 > p0 ? (p1 - p0 + BN - 1) / BN : 0;

    auto load_kv = [&](int tile, int stage) {
        const int v0 = p0 + tile * BN, n0 = v0 < front ? v0 : v0 + shift;
        __half* dk = sK + stage * BN * LD;
        __half* dv = sV + stage * BN * LD;
        const size_t r0 = paged_row(a.page_table + (size_t)slot * a.max_pages, n0, a.n_kv_heads, kvh);
        for (int c = tid; c < BN * (D / 8); c += 128) {
            const int r = c / (D / 8), col = (c % (D / 8)) * 8;
            cp_async16(dk + r * LD + col, a.k_cache + (r0 + r) * D + col);
            cp_async16(dv + r * LD + col, a.v_cache + (r0 + r) * D + col);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // the first NS - 1 tiles are requested at once (one commit group each, empty past the end, so that the counting stays uniform)
#pragma unroll
    for (int t = 0; t < NS - 1; t++) {
        if (t < n_tiles) load_kv(t, t);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
        const bool owner = !r.no_append && n_tiles > 0 && qpos - shift >= p0 && qpos - shift < p1;      // this split holds the query token's own position
    // element i of a raw head row after the rotary embedding (pairs (2p, 2p+1), or (p, p + n_rot/2) in the neox order)
    // the second map's columns of a row of two (differential attention) turn like the first's
    auto rotated = [&](const float* row, int i) -> float {
        const float x = row[i];
        if (r.maps > 1 && i >= r.dim) {
            i -= r.dim;
            row += r.dim;
            if (i >= r.dim) return x;
        }
        if (i >= r.n_rot) return x;
        const int half_rot = r.n_rot >> 1;
        const bool first = r.neox ? i < half_rot : !(i & 1);
        const int p = r.neox ? (first ? i : i - half_rot) : i >> 1;
        const float y = row[r.neox ? (first ? i + half_rot : i - half_rot) : (i ^ 1)];
        return first ? x * s_cs[p] - y * s_sn[p] : y * s_sn[p] + x * s_cs[p];
    };
    {
        // the raw rows (query heads of this group, the key and the value) are staged in the last K stage, which stays unused
        // until the tile loop requests tile NS - 1; cos / sin of the position are computed once per CTA meanwhile
        float* raw = reinterpret_cast<float*>(sK + (TS - 1) * BN * LD);       // [group + 2][D]
        const int nrows = group + (owner ? 2 : 0);
        const float* tok = r.qkv + (size_t)b * r.ldq;
        const int kdim = r.maps * r.dim, nq = a.n_heads * r.dim, nk = a.n_kv_heads * kdim;
        for (int p = tid; p < (r.n_rot >> 1); p += 128) {
            float sn, cs;
            sincosf(rot_angle(qpos, r.freqs[p]), &sn, &cs);
            s_sn[p] = sn * r.mscale;
            s_cs[p] = cs * r.mscale;
        }
        float iq = 1.f, ik = 1.f;
        if (r.q_norm && !r.head_norm) {
            float s0 = 0.f, s1 = 0.f;
            const int total = owner ? nq + nk : nq;
            if (((nq | nk | r.ldq) & 3) == 0) {
#pragma unroll 8
                for (int i = 4 * tid; i < total; i += 512) {
                    const float4 v = __ldcg(reinterpret_cast<const float4*>(tok + i));
                    const float d = v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
                    if (i < nq) s0 += d;
                    else s1 += d;
                }
            } else {
                for (int i = tid; i < total; i += 128) {
                    const float d = tok[i] * tok[i];
                    if (i < nq) s0 += d;
                    else s1 += d;
                }
            }
            s0 = warp_sum(s0);
            s1 = warp_sum(s1);
            if (lane == 0) {
                s_m[warp][0] = s0;
                s_l[warp][0] = s1;
            }
            __syncthreads();
            iq = 1.f / sqrtf((s_m[0][0] + s_m[1][0] + s_m[2][0] + s_m[3][0]) / (float)nq + r.eps);
            ik = 1.f / sqrtf((s_l[0][0] + s_l[1][0] + s_l[2][0] + s_l[3][0]) / (float)nk + r.eps);
        }
#pragma unroll 4
        for (int c = tid; c < nrows * D; c += 128) {
            const int rr = c / D, col = c % D;
            float v = 0.f;
            if (rr <= group) {
                const int off = rr < group ? (head0 + rr) % r.maps * r.dim : 0;
                if (col >= off && col < (rr < group ? off + r.dim : kdim)) {
                    const int i = rr < group ? (head0 + rr) * r.dim + col - off : kvh * kdim + col;
                    v = tok[rr < group ? i : nq + i];
                    if (r.q_norm && !r.head_norm) v *= rr < group ? iq * r.q_norm[i] : ik * r.k_norm[i];
                }
            } else if (col < r.vdim) {
                v = tok[r.v_off + kvh * r.vdim + col];
            }
            raw[c] = v;
        }
        if (r.q_norm && r.head_norm) {          // a warp per head
            __syncthreads();
            for (int rr = warp; rr < group + (owner ? 1 : 0); rr += 4) {
                const float* w = rr < group ? r.q_norm : r.k_norm;
                float x[D / 32], s = 0.f;
#pragma unroll
                for (int i = 0; i < D / 32; i++) {
                    x[i] = raw[rr * D + lane + 32 * i];      // columns beyond dim are zero
                    s += x[i] * x[i];
                }
                const float inv = 1.f / sqrtf(warp_sum(s) / (float)r.dim + r.eps);
#pragma unroll
                for (int i = 0; i < D / 32; i++)
                    if (lane + 32 * i < r.dim) raw[rr * D + lane + 32 * i] = x[i] * inv * w[lane + 32 * i];
            }
        }
        __syncthreads();
        if (owner) {      // append the new key / value rows to the cache and keep them for the last tile
            const float* krow = raw + group * D;
            const float* vrow = raw + (group + 1) * D;
            const size_t own = paged_row(a.page_table + (size_t)slot * a.max_pages, qpos, a.n_kv_heads, kvh);
            __half* kc = const_cast<__half*>(a.k_cache) + own * D;
            __half* vc = const_cast<__half*>(a.v_cache) + own * D;
            for (int i = tid; i < D; i += 128) {
                const __half kh = __float2half_rn(rotated(krow, i)), vh = __float2half_rn(vrow[i]);
                s_newk[i] = kh;
                s_newv[i] = vh;
                kc[i] = kh;
                vc[i] = vh;
            }
        }
        for (int c = tid; c < ROWS * (D / 4); c += 128) {
            const int rr = c / (D / 4), col = (c % (D / 4)) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (rr < group) {
                const float* qrow = raw + rr * D;
                v = make_float4(rotated(qrow, col), rotated(qrow, col + 1), rotated(qrow, col + 2), rotated(qrow, col + 3));
            }
            *reinterpret_cast<uint2*>(sQ + rr * LD + col) = make_uint2(pack_half2(v.x, v.y), pack_half2(v.z, v.w));
        }
    }
    __syncthreads();
    uint32_t qf[D / 16][4];
#pragma unroll
    for (int kk = 0; kk < D / 16; kk++)
        ldmatrix_x4(qf[kk], smem_addr(sQ + ((lane & 7) + 8 * ((lane >> 3) & 1)) * LD + kk * 16 + 8 * (lane >> 4)));

    float o[D / 8][4];
#pragma unroll
    for (int j = 0; j < D / 8; j++) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    float m_run[2] = {-1e30f, -1e30f}, l_run[2] = {0.f, 0.f};
    const float inv_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;

    for (int tile = 0; tile < n_tiles; tile++) {
        const int stage = tile % NS;
        if (tile + NS - 1 < n_tiles) load_kv(tile + NS - 1, (tile + NS - 1) % NS);      // into the stage that tile - 1 has just left
        else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group %0;" ::"n"(NS - 1) : "memory");               // tile's own group is complete
        __syncthreads();
        if (owner && tile == n_tiles - 1) {      // the query's own row did not come from the cache: put it into the tile
            const int rr = qpos - shift - (p0 + tile * BN);
            for (int i = tid; i < D; i += 128) {
                sK[stage * BN * LD + rr * LD + i] = s_newk[i];
                sV[stage * BN * LD + rr * LD + i] = s_newv[i];
            }
            __syncthreads();
        }
        const __half* tk = sK + stage * BN * LD + 16 * warp * LD;       // this warp's 16 positions of the tile
        const __half* tv = sV + stage * BN * LD + 16 * warp * LD;
        const int v0 = p0 + tile * BN, n0 = (v0 < front ? v0 : v0 + shift) + 16 * warp, end = v0 < front ? n0 + BN : p1 + shift;

        float s[2][4];
        s[0][0] = s[0][1] = s[0][2] = s[0][3] = s[1][0] = s[1][1] = s[1][2] = s[1][3] = 0.f;
#pragma unroll
        for (int kk = 0; kk < D / 16; kk++) {
            uint32_t kb[4];
            ldmatrix_x4(kb, smem_addr(tk + ((lane & 7) + 8 * (lane >> 4)) * LD + kk * 16 + 8 * ((lane >> 3) & 1)));
            mma_f16(s[0], qf[kk], kb[0], kb[1]);
            mma_f16(s[1], qf[kk], kb[2], kb[3]);
        }
        // element e of block j: row g + 8 (e >> 1) (a query head), position n0 + 8 j + 2 tq + (e & 1)
        float mx[2] = {-1e30f, -1e30f};
        bool ok[2][2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int kp = n0 + 8 * j + 2 * tq + e;
                ok[j][e] = kp < end && (kp >= start || kp < keep);
            }
#pragma unroll
            for (int e = 0; e < 4; e++) {
                float v = s[j][e] * a.scale;
                if (a.softcap > 0.f) v = a.softcap * tanh_exp(v * inv_cap);
                s[j][e] = v;
                if (ok[j][e & 1]) mx[e >> 1] = fmaxf(mx[e >> 1], v);
            }
        }
        float corr[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
            const float m_new = fmaxf(m_run[r], mx[r]);
            corr[r] = __expf(m_run[r] - m_new);
            m_run[r] = m_new;
            l_run[r] *= corr[r];
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float p = ok[j][e & 1] ? __expf(s[j][e] - m_run[e >> 1]) : 0.f;
                s[j][e] = p;
                l_run[e >> 1] += p;
            }
        }
#pragma unroll
        for (int j = 0; j < D / 8; j++) {
            o[j][0] *= corr[0]; o[j][1] *= corr[0];
            o[j][2] *= corr[1]; o[j][3] *= corr[1];
        }
        // O += P V: the accumulator fragments of S are the A fragments of P (16 positions = one k step)
        uint32_t pa[4];
        pa[0] = pack_half2(s[0][0], s[0][1]);
        pa[1] = pack_half2(s[0][2], s[0][3]);
        pa[2] = pack_half2(s[1][0], s[1][1]);
        pa[3] = pack_half2(s[1][2], s[1][3]);
#pragma unroll
        for (int j = 0; j < D / 8; j += 2) {
            uint32_t vb[4];
            ldmatrix_x4_trans(vb, smem_addr(tv + ((lane & 7) + 8 * ((lane >> 3) & 1)) * LD + 8 * j + 8 * (lane >> 4)));
            mma_f16(o[j], pa, vb[0], vb[1]);
            mma_f16(o[j + 1], pa, vb[2], vb[3]);
        }
        __syncthreads();        // everyone is done with this stage before the next iteration's request overwrites it
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    // merge the four warps: (max, sum, acc) of every query head through shared memory (the staging area is free now)
#pragma unroll
    for (int r = 0; r < 2; r++) {
        l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
        l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
    }
    float* s_acc = reinterpret_cast<float*>(sK);                 // [4][ROWS][D]
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int row = g + 8 * r;
        if (row < group) {
            float* dst = s_acc + ((size_t)warp * ROWS + row) * D;
#pragma unroll
            for (int j = 0; j < D / 8; j++) *reinterpret_cast<float2*>(dst + 8 * j + 2 * tq) = make_float2(o[j][2 * r], o[j][2 * r + 1]);
            if (tq == 0) {
                s_m[warp][row] = m_run[r];
                s_l[warp][row] = l_run[r];
            }
        }
    }
    __syncthreads();
    for (int idx = tid; idx < group * D; idx += 128) {
        const int row = idx / D, d = idx % D;
        const float mn = fmaxf(fmaxf(s_m[0][row], s_m[1][row]), fmaxf(s_m[2][row], s_m[3][row]));
        float acc = 0.f, lt = 0.f;
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const float c = __expf(s_m[w][row] - mn);
            acc += s_acc[((size_t)w * ROWS + row) * D + d] * c;
            lt += s_l[w][row] * c;
        }
        const size_t pi = ((size_t)b * a.n_heads + head0 + row) * a.n_splits + split;
        a.part_acc[pi * D + d] = acc;
        if (d == 0) a.part_ml[pi] = make_float2(mn, lt);
    }
}


// Flat caches: every warp streams 16 positions at a time through a ring of its own, so that nothing in the loop waits for another warp (tiles of 64 positions that the four
// warps shared cost two or three barriers each; with what their int8 form expanded in between, 8 sequences of 3000 positions took 34 us a layer for 8 us of bytes).
// The positions of all sequences of a launch are dealt out to about as many CTAs as fit the GPU at once (`room` of them a KV head, 0: every sequence to all its splits), each an
// equal share of one sequence; what is left of a sequence's splits only says that it is empty.  With the merge, us a layer (32 heads of 128 on 8): 8 sequences about 3000, int8
// 35.2 -> 23.2, f16 29.2 -> 26.0 (bytes 15); 32 about 467 22.3 -> 20.6 (bytes 9.3), with sixteen splits allocated 34.6 -> 22.2; 64 heads of 64, 16 about 1024 18.3 -> 15.9.
// What is left: three CTAs of four warps an SM (registers) whose turn takes about as long as its rows, the launch, the first rows' latency and the merge (6 us).
// Q8: rows stay int8 in the ring.  A key word (four dims) becomes two B-fragment registers in place, which is why the queries' fragments have a lane's dims in that order;
// values are expanded into a tile of the warp's own.  With raw projections the owning split quantises the new rows as b2_rope_kv does, instead of that launch before this one: a step of 8
// sequences of 12 layers 1096 -> 1073 us.
template <int D, int NS, bool Q8>
__global__ void __launch_bounds__(128) attn_decode_flat_kernel(const __grid_constant__ AttnDecodeArgs a, const __grid_constant__ AttnRopeArgs r, int room) {
    constexpr int LD = D + PAD, NW = 16;                          // positions of a warp's turn
    constexpr int SCALES = NW * D / 16;                           // bytes of a turn's scales of keys or values
    constexpr int STAGE = Q8 ? 2 * (NW * D + SCALES) : 2 * NW * LD * 2, WIDE = Q8 ? NW * LD * 2 : 0;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __half* sQ = reinterpret_cast<__half*>(smem_raw);            // [ROWS][LD]
    __shared__ float s_m[4][ROWS], s_l[4][ROWS];
    __shared__ float s_cs[128], s_sn[128];                        // cos / sin of the query position per rotated pair (fused form)
    __shared__ __half s_newk[D], s_newv[D];                       // the query token's own key and value rows (fused form, owning split)
    __shared__ int8_t s_new8[2][D];                               // Q8: their codes, whose scales are s_newk[i], s_newv[i] of dims 32 i ..
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
    unsigned char* ring = smem_raw + ROWS * LD * 2 + warp * (NS * STAGE + WIDE);
    __half* wide = reinterpret_cast<__half*>(ring + NS * STAGE);  // Q8: [NW][LD] values
    const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
    const int group = a.n_heads / a.n_kv_heads;                  // query heads per KV head (<= ROWS, checked by the launcher)
    const int head0 = kvh * group;

    pdl_launch();
    pdl_wait();
    const int qpos = a.positions[b], slot = a.slots[b];
    const int kv_len = qpos + 1, start = first_key(qpos, 0, a.window), span = kv_len - start;
    int chunk = (span + a.n_splits - 1) / a.n_splits;
    if (room > 0) {
        int sum = 0, longest = 0;
        for (int i = lane; i < (int)gridDim.z; i += 32) {
            const int p = a.positions[i], n = p + 1 - first_key(p, 0, a.window);
            sum += n;
            longest = max(longest, n);
        }
        sum = __reduce_add_sync(0xffffffffu, sum);
        longest = __reduce_max_sync(0xffffffffu, longest);
        // ceil(n / chunk) of all sequences: at most sum / chunk + their number
        chunk = max((sum + room - (int)gridDim.z - 1) / (room - (int)gridDim.z), (longest + a.n_splits - 1) / a.n_splits);
    }
    chunk = ((chunk + BN - 1) / BN) * BN;
    const int p0 = start + split * chunk, p1 = min(p0 + chunk, kv_len);
    if (p0 >= p1) {      // nothing left for this split: the combine kernel skips it
        if (tid < group) a.part_ml[((size_t)b * a.n_heads + head0 + tid) * a.n_splits + split] = make_float2(-1e30f, 0.f);
        return;
    }
    const size_t row0 = ((size_t)slot * a.n_kv_heads + kvh) * a.n_ctx;      // first cache row of this (slot, kv head)
    const int turns = (p1 - p0 - NW * warp + 4 * NW - 1) / (4 * NW);        // this warp has positions p0 + 16 (warp + 4 i) ..

    auto request = [&](int i) {      // rows past the range repeat a valid row (masked below)
        if (i < turns) {
            const int n0 = p0 + NW * (warp + 4 * i);
            unsigned char* to = ring + i % NS * STAGE;
            if (Q8) {
#pragma unroll
                for (int kv = 0; kv < 2; kv++) {
                    const unsigned char* from = reinterpret_cast<const unsigned char*>(kv ? a.v_cache : a.k_cache) + row0 * D;
                    const __half* sc = (kv ? a.v_scale : a.k_scale) + row0 * (D / 32);
#pragma unroll
                    for (int c = lane; c < NW * (D / 16); c += 32) {      // 16-byte pieces; of rows of 128 bytes odd ones have their halves exchanged
                        const int rr = c / (D / 16), piece = c % (D / 16);
                        cp_async16(to + rr * D + ((D == 128 ? piece ^ (4 * (rr & 1)) : piece) << 4), from + (size_t)min(n0 + rr, a.n_ctx - 1) * D + 16 * piece);
                    }
                    if (lane < NW) {      // the row's scales: D / 16 bytes
                        const __half* at = sc + (size_t)min(n0 + lane, a.n_ctx - 1) * (D / 32);
                        unsigned char* sto = to + NW * D + lane * (D / 16);
                        if (D == 128) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(sto)), "l"(at) : "memory");
                        else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(sto)), "l"(at) : "memory");
                    }
                    to += NW * D + SCALES;
                }
            } else {
                __half* dk = reinterpret_cast<__half*>(to);
                __half* dv = dk + NW * LD;
#pragma unroll
                for (int c = lane; c < NW * (D / 8); c += 32) {
                    const int rr = c / (D / 8), col = (c % (D / 8)) * 8;
                    const size_t at = (row0 + min(n0 + rr, a.n_ctx - 1)) * D + col;
                    cp_async16(dk + rr * LD + col, a.k_cache + at);
                    cp_async16(dv + rr * LD + col, a.v_cache + at);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the first NS - 1 turns are requested at once (one commit group each, empty past the end, so that the counting stays uniform)
#pragma unroll
    for (int i = 0; i < NS - 1; i++) request(i);

    const bool fresh = r.qkv != nullptr;
    const bool owner = fresh && qpos >= p0 && qpos < p1;          // this split holds the query token's own position
    // element i of a raw head row after the rotary embedding (pairs (2p, 2p+1), or (p, p + n_rot/2) in the neox order)
    auto rotated = [&](const float* row, int i) -> float {
        const float x = row[i];
        if (i >= r.n_rot) return x;
        const int half_rot = r.n_rot >> 1;
        const bool first = r.neox ? i < half_rot : !(i & 1);
        const int p = r.neox ? (first ? i : i - half_rot) : i >> 1;
        const float y = row[r.neox ? (first ? i + half_rot : i - half_rot) : (i ^ 1)];
        return first ? x * s_cs[p] - y * s_sn[p] : y * s_sn[p] + x * s_cs[p];
    };
    if (fresh) {
        // the raw rows (query heads of this group, the key and the value) are staged from the last warp's last stage on, which no request has reached yet; cos / sin of the
        // position are computed once per CTA meanwhile
        float* raw = reinterpret_cast<float*>(smem_raw + ROWS * LD * 2 + 3 * (NS * STAGE + WIDE) + (NS - 1) * STAGE);       // [group + 2][D]
        const int nrows = group + (owner ? 2 : 0);
        const float* tok = r.qkv + (size_t)b * (a.n_heads + 2 * a.n_kv_heads) * D;
        for (int c = tid; c < nrows * (D / 4); c += 128) {
            const int rr = c / (D / 4), col = (c % (D / 4)) * 4;
            const float* src = rr < group ? tok + (size_t)(head0 + rr) * D
                                          : tok + (size_t)(a.n_heads + (rr == group ? 0 : a.n_kv_heads) + kvh) * D;
            *reinterpret_cast<float4*>(raw + rr * D + col) = __ldcg(reinterpret_cast<const float4*>(src + col));
        }
        for (int p = tid; p < (r.n_rot >> 1); p += 128) {
            float sn, cs;
            sincosf((float)qpos * r.inv_freq[p], &sn, &cs);
            s_sn[p] = sn * r.mscale;
            s_cs[p] = cs * r.mscale;
        }
        if (r.q_norm) {          // RMS norm of each head, a warp per head
            __syncthreads();
            for (int rr = warp; rr < group + (owner ? 1 : 0); rr += 4) {
                const float* w = rr < group ? r.q_norm : r.k_norm;
                float x[D / 32], s = 0.f;
#pragma unroll
                for (int i = 0; i < D / 32; i++) {
                    x[i] = raw[rr * D + lane + 32 * i];
                    s += x[i] * x[i];
                }
                const float inv = rsqrtf(warp_sum(s) / (float)D + r.eps);
#pragma unroll
                for (int i = 0; i < D / 32; i++) raw[rr * D + lane + 32 * i] = x[i] * inv * w[lane + 32 * i];
            }
        }
        __syncthreads();
        if (owner) {      // append the new key / value rows to the cache and keep them for the turn that holds their position
            const float* krow = raw + group * D;
            const float* vrow = raw + (group + 1) * D;
            __half* kc = const_cast<__half*>(a.k_cache) + (row0 + qpos) * D;
            __half* vc = const_cast<__half*>(a.v_cache) + (row0 + qpos) * D;
            for (int i = tid; i < D; i += 128) {
                const float k = rotated(krow, i), v = vrow[i];
                if (Q8) {      // a warp has a block of 32 dims
                    const __half hk = __float2half_rn(warp_max(fabsf(k)) / 127.f), hv = __float2half_rn(warp_max(fabsf(v)) / 127.f);
                    const float dk = __half2float(hk), dv = __half2float(hv);
                    const int8_t qk = (int8_t)(dk > 0.f ? max(-127, min(127, __float2int_rn(k / dk))) : 0), qv = (int8_t)(dv > 0.f ? max(-127, min(127, __float2int_rn(v / dv))) : 0);
                    s_new8[0][i] = qk;
                    s_new8[1][i] = qv;
                    const_cast<int8_t*>(reinterpret_cast<const int8_t*>(a.k_cache))[(row0 + qpos) * D + i] = qk;
                    const_cast<int8_t*>(reinterpret_cast<const int8_t*>(a.v_cache))[(row0 + qpos) * D + i] = qv;
                    if (lane == 0) {
                        const size_t at = (row0 + qpos) * (D / 32) + (i >> 5);
                        const_cast<__half*>(a.k_scale)[at] = s_newk[i >> 5] = hk;
                        const_cast<__half*>(a.v_scale)[at] = s_newv[i >> 5] = hv;
                    }
                    continue;
                }
                const __half kh = __float2half_rn(k), vh = __float2half_rn(v);
                s_newk[i] = kh;
                s_newv[i] = vh;
                kc[i] = kh;
                vc[i] = vh;
            }
        }
        for (int c = tid; c < ROWS * (D / 4); c += 128) {
            const int rr = c / (D / 4), col = (c % (D / 4)) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (rr < group) {
                const float* qrow = raw + rr * D;
                v = make_float4(rotated(qrow, col), rotated(qrow, col + 1), rotated(qrow, col + 2), rotated(qrow, col + 3));
            }
            *reinterpret_cast<uint2*>(sQ + rr * LD + col) = make_uint2(pack_half2(v.x, v.y), pack_half2(v.z, v.w));
        }
    } else {
        // Q rows: the heads of this KV head, fp32 -> f16, rows beyond the group are zero
        for (int c = tid; c < ROWS * (D / 4); c += 128) {
            const int rr = c / (D / 4), col = (c % (D / 4)) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (rr < group) v = *(const float4*)(a.q + ((size_t)b * a.n_heads + head0 + rr) * D + col);
            *reinterpret_cast<uint2*>(sQ + rr * LD + col) = make_uint2(pack_half2(v.x, v.y), pack_half2(v.z, v.w));
        }
    }
    __syncthreads();
    uint32_t qf[D / 16][4];
#pragma unroll
    for (int kk = 0; kk < D / 16; kk++) {
        if (Q8) {      // product kk takes dims 64 (kk / 4) + 16 tq + 4 (kk & 3) .. + 3 of lane tq
            const int col = 64 * (kk >> 2) + 16 * tq + 4 * (kk & 3);
            const uint2 lo = *reinterpret_cast<const uint2*>(sQ + g * LD + col), hi = *reinterpret_cast<const uint2*>(sQ + (g + 8) * LD + col);
            qf[kk][0] = lo.x; qf[kk][1] = hi.x; qf[kk][2] = lo.y; qf[kk][3] = hi.y;
        } else {
            ldmatrix_x4(qf[kk], smem_addr(sQ + ((lane & 7) + 8 * ((lane >> 3) & 1)) * LD + kk * 16 + 8 * (lane >> 4)));
        }
    }

    float o[D / 8][4];
#pragma unroll
    for (int j = 0; j < D / 8; j++) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    float m_run[2] = {-1e30f, -1e30f}, l_run[2] = {0.f, 0.f};
    const float inv_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;

    for (int i = 0; i < turns; i++) {
        request(i + NS - 1);                                                             // into the stage of the turn before
        asm volatile("cp.async.wait_group %0;" ::"n"(NS - 1) : "memory");
        __syncwarp();
        unsigned char* st = ring + i % NS * STAGE;
        const int n0 = p0 + NW * (warp + 4 * i);
        __half* tk = reinterpret_cast<__half*>(st);
        const __half* tv = Q8 ? wide : tk + NW * LD;
        if (owner && n0 <= qpos && qpos < n0 + NW) {      // the query's own row did not come from the cache
            const int rr = qpos - n0;
            __half* dk = tk + rr * LD;
            for (int d = lane; d < D; d += 32) {
                if (Q8) {
                    unsigned char* to = st + rr * D + ((D == 128 ? (d >> 4) ^ (4 * (rr & 1)) : d >> 4) << 4) + (d & 15);
                    to[0] = (unsigned char)s_new8[0][d];
                    to[NW * D + SCALES] = (unsigned char)s_new8[1][d];
                } else {
                    dk[d] = s_newk[d];
                    dk[NW * LD + d] = s_newv[d];
                }
            }
            if (Q8 && lane < D / 32) {
                __half* sc = reinterpret_cast<__half*>(st + NW * D) + rr * (D / 32) + lane;
                sc[0] = s_newk[lane];
                sc[(NW * D + SCALES) / 2] = s_newv[lane];
            }
            __syncwarp();
        }
        float s[2][4];
        s[0][0] = s[0][1] = s[0][2] = s[0][3] = s[1][0] = s[1][1] = s[1][2] = s[1][3] = 0.f;
        if (Q8) {
            const __half* ksc = reinterpret_cast<const __half*>(st + NW * D);
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int h = 0; h < D / 64; h++) {
                    const int rr = 8 * j + g, piece = 4 * h + tq;
                    const uint4 w = *reinterpret_cast<const uint4*>(st + rr * D + ((D == 128 ? piece ^ (4 * (rr & 1)) : piece) << 4));
                    const __half2 d = __half2half2(ksc[rr * (D / 32) + 2 * h + (tq >> 1)]);
                    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const uint2 e = expand_q8x4(u[q], d);
                        mma_f16(s[j], qf[4 * h + q], e.x, e.y);
                    }
                }
            // values to f16
            const unsigned char* vst = st + NW * D + SCALES;
            const __half* vsc = reinterpret_cast<const __half*>(vst + NW * D);
#pragma unroll
            for (int c = lane; c < NW * (D / 16); c += 32) {
                const int rr = c / (D / 16), piece = c % (D / 16);
                const uint4 w = *reinterpret_cast<const uint4*>(vst + rr * D + ((D == 128 ? piece ^ (4 * (rr & 1)) : piece) << 4));
                const __half2 d = __half2half2(vsc[rr * (D / 32) + (piece >> 1)]);
                const uint2 e0 = expand_q8x4(w.x, d), e1 = expand_q8x4(w.y, d), e2 = expand_q8x4(w.z, d), e3 = expand_q8x4(w.w, d);
                *reinterpret_cast<uint4*>(wide + rr * LD + 16 * piece) = make_uint4(e0.x, e0.y, e1.x, e1.y);
                *reinterpret_cast<uint4*>(wide + rr * LD + 16 * piece + 8) = make_uint4(e2.x, e2.y, e3.x, e3.y);
            }
            __syncwarp();
        } else {
#pragma unroll
            for (int kk = 0; kk < D / 16; kk++) {
                uint32_t kb[4];
                ldmatrix_x4(kb, smem_addr(tk + ((lane & 7) + 8 * (lane >> 4)) * LD + kk * 16 + 8 * ((lane >> 3) & 1)));
                mma_f16(s[0], qf[kk], kb[0], kb[1]);
                mma_f16(s[1], qf[kk], kb[2], kb[3]);
            }
        }
        // element e of block j: row g + 8 (e >> 1) (a query head), position n0 + 8 j + 2 tq + (e & 1)
        float mx[2] = {-1e30f, -1e30f};
        bool ok[2][2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
#pragma unroll
            for (int e = 0; e < 2; e++) ok[j][e] = n0 + 8 * j + 2 * tq + e < p1;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                float v = s[j][e] * a.scale;
                if (a.softcap > 0.f) v = a.softcap * tanh_exp(v * inv_cap);
                s[j][e] = v;
                if (ok[j][e & 1]) mx[e >> 1] = fmaxf(mx[e >> 1], v);
            }
        }
        float corr[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], 1));
            mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], 2));
            const float m_new = fmaxf(m_run[q], mx[q]);
            corr[q] = __expf(m_run[q] - m_new);
            m_run[q] = m_new;
            l_run[q] *= corr[q];
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float p = ok[j][e & 1] ? __expf(s[j][e] - m_run[e >> 1]) : 0.f;
                s[j][e] = p;
                l_run[e >> 1] += p;
            }
        }
#pragma unroll
        for (int j = 0; j < D / 8; j++) {
            o[j][0] *= corr[0]; o[j][1] *= corr[0];
            o[j][2] *= corr[1]; o[j][3] *= corr[1];
        }
        // O += P V: the accumulator fragments of S are the A fragments of P (16 positions = one k step)
        uint32_t pa[4];
        pa[0] = pack_half2(s[0][0], s[0][1]);
        pa[1] = pack_half2(s[0][2], s[0][3]);
        pa[2] = pack_half2(s[1][0], s[1][1]);
        pa[3] = pack_half2(s[1][2], s[1][3]);
#pragma unroll
        for (int j = 0; j < D / 8; j += 2) {
            uint32_t vb[4];
            ldmatrix_x4_trans(vb, smem_addr(tv + ((lane & 7) + 8 * ((lane >> 3) & 1)) * LD + 8 * j + 8 * (lane >> 4)));
            mma_f16(o[j], pa, vb[0], vb[1]);
            mma_f16(o[j + 1], pa, vb[2], vb[3]);
        }
        __syncwarp();        // every lane is done with this stage before the next turn's request overwrites it
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    // merge the four warps: (max, sum, acc) of every query head through shared memory (behind the barrier the rings are free)
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; q++) {
        l_run[q] += __shfl_xor_sync(0xffffffffu, l_run[q], 1);
        l_run[q] += __shfl_xor_sync(0xffffffffu, l_run[q], 2);
    }
    float* s_acc = reinterpret_cast<float*>(smem_raw + ROWS * LD * 2);                 // [4][ROWS][D]
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int row = g + 8 * q;
        if (row < group) {
            float* dst = s_acc + ((size_t)warp * ROWS + row) * D;
#pragma unroll
            for (int j = 0; j < D / 8; j++) *reinterpret_cast<float2*>(dst + 8 * j + 2 * tq) = make_float2(o[j][2 * q], o[j][2 * q + 1]);
            if (tq == 0) {
                s_m[warp][row] = m_run[q];
                s_l[warp][row] = l_run[q];
            }
        }
    }
    __syncthreads();
    for (int idx = tid; idx < group * D; idx += 128) {
        const int row = idx / D, d = idx % D;
        const float mn = fmaxf(fmaxf(s_m[0][row], s_m[1][row]), fmaxf(s_m[2][row], s_m[3][row]));
        float acc = 0.f, lt = 0.f;
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const float c = __expf(s_m[w][row] - mn);
            acc += s_acc[((size_t)w * ROWS + row) * D + d] * c;
            lt += s_l[w][row] * c;
        }
        const size_t pi = ((size_t)b * a.n_heads + head0 + row) * a.n_splits + split;
        a.part_acc[pi * D + d] = acc;
        if (d == 0) a.part_ml[pi] = make_float2(mn, lt);
    }
}

int sm_count() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    return sms;
}

// room: of the flat kernel, negative: the paged one
int start(const void* fn, int smem, const AttnDecodeArgs& a, const AttnRopeArgs& r, int nb, int room, int pdl, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.n_splits, a.n_kv_heads, nb);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    AttnDecodeArgs copy = a;
    AttnRopeArgs rcopy = r;
    void* args[] = {&copy, &rcopy, &room};
    return (int)cudaLaunchKernelExC(&cfg, fn, args);
}

template <int D, int NS>
int launch_paged(const AttnDecodeArgs& a, const AttnRopeArgs& r, int nb, int pdl, cudaStream_t st) {
    constexpr int SMEM = (ROWS + 2 * NS * BN) * (D + PAD) * 2;
    const void* fn = (const void*)attn_decode_paged_kernel<D, NS>;
    static PerDeviceOnce once;
    if (once.first()) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    return start(fn, SMEM, a, r, nb, -1, pdl, st);
}

template <int D, int NS, bool Q8 = false>
int launch_flat(const AttnDecodeArgs& a, const AttnRopeArgs& r, int nb, int pdl, cudaStream_t st) {
    constexpr int WARP = Q8 ? NS * 2 * (16 * D + D) + 16 * (D + PAD) * 2 : NS * 2 * 16 * (D + PAD) * 2;
    constexpr int RINGS = ROWS * (D + PAD) * 2 + 4 * WARP, MERGE = ROWS * (D + PAD) * 2 + 4 * ROWS * D * 4;
    constexpr int LAST = Q8 ? 2 * 17 * D + 16 * (D + PAD) * 2 : WARP / NS;                        // the last warp's last stage and what lies behind it
    const int raw = r.qkv ? RINGS - LAST + (a.n_heads / a.n_kv_heads + 2) * D * 4 : 0;            // where the raw rows end
    int smem = RINGS > MERGE ? RINGS : MERGE;
    if (raw > smem) smem = raw;
    const void* fn = (const void*)attn_decode_flat_kernel<D, NS, Q8>;
    static PerDeviceOnce once;
    if (once.first()) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (RINGS > MERGE ? RINGS : MERGE) + (ROWS + 2) * D * 4);
    // Launches of more CTAs than fit at once deal the positions out to as many as do; MHA steps that have more sequences and heads than that keep about two a sequence.
    const int per_sm = 228 * 1024 / (smem + 3 * 1024), fit = per_sm * sm_count() / a.n_kv_heads;
    const int room = (long)a.n_splits * nb <= fit ? 0 : fit > 2 * nb ? fit : 2 * nb;
    return start(fn, smem, a, r, nb, room, pdl, st);
}

int g_stages = 0;      // 0: by the size of the launch; 2, 3 or 4: forced (tests)

// Four stages take 140 KB of shared memory (one CTA per SM), three 109 KB (two per SM), two 74 KB (three per SM).  A launch that
// gives every SM at most one CTA runs four stages, one that gives it at most two runs three, larger ones keep two: the bytes in
// flight per SM stay about the same and no launch needs a second round because of its shared memory.
// int8 caches take 91 KB in four stages and 74 KB, three CTAs per SM, in three, their least.  Steps of at most one CTA per SM in three and in four stages: Llama-8B, one sequence, 4 layers of
// Q8_0 433 and 412 us at 400 positions, 455 and 430 at 4000, 12 layers of Q4_K_M 666 and 660, 733 and 715 (at 60 663 and 666); 20 layers of 16 heads on 4, two sequences about 4000 1241
// and 1171.
int stages_for(const AttnDecodeArgs& a, int nb) {
    int ns = g_stages;
    if (!ns) {
        const long ctas = (long)a.n_splits * a.n_kv_heads * nb;
        ns = a.n_ctx / a.n_splits < 2 * BN ? 2 : ctas <= sm_count() ? 4 : ctas <= 2L * sm_count() ? 3 : 2;
    }
    return a.k_scale && ns < 3 ? 3 : ns;
}

template <int D>
int launch_d(const AttnDecodeArgs& a, const AttnRopeArgs& r, int nb, int pdl, cudaStream_t st) {
    const int ns = stages_for(a, nb);
    if (a.page_table) return ns == 4 ? launch_paged<D, 4>(a, r, nb, pdl, st) : ns == 3 ? launch_paged<D, 3>(a, r, nb, pdl, st) : launch_paged<D, 2>(a, r, nb, pdl, st);
    if (a.k_scale) return ns == 4 ? launch_flat<D, 4, true>(a, r, nb, pdl, st) : launch_flat<D, 3, true>(a, r, nb, pdl, st);
    return ns == 4 ? launch_flat<D, 4>(a, r, nb, pdl, st) : ns == 3 ? launch_flat<D, 3>(a, r, nb, pdl, st) : launch_flat<D, 2>(a, r, nb, pdl, st);
}

}  // namespace

// 1 if the tensor-core kernel takes caches like these, 0 if the scalar one has to (nothing is launched).  A row's int8 scales are fetched at once, hd / 16 bytes of them.
B2_API int b2_attn_decode_mma_takes(const AttnDecodeArgs* a, int hd) {
    if (hd != 64 && hd != 128) return 0;
    if (a->n_kv_heads < 1 || a->n_heads % a->n_kv_heads || a->n_heads / a->n_kv_heads > ROWS) return 0;
    return !a->k_scale || !(((uintptr_t)a->k_scale | (uintptr_t)a->v_scale) & (hd / 16 - 1));
}

// Splits of a sequence that a launch on flat caches uses: a step of many sequences fills the GPU with few of them, and every CTA that finds nothing to do costs its launch (32
// sequences, 16 splits: 35 us a layer for what 7 splits do in 21).
int attn_decode_mma_splits(const AttnDecodeArgs& a, int nb) {
    if (a.page_table) return a.n_splits;
    const int most = 4 * 3 * sm_count() / (a.n_kv_heads * nb) + 1;
    return most < 4 ? (a.n_splits < 4 ? a.n_splits : 4) : most < a.n_splits ? most : a.n_splits;
}

int attn_decode_mma_rope_launch(const AttnDecodeArgs& a, const AttnRopeArgs& r, int nb, int hd, int pdl, cudaStream_t st) {
    if (!b2_attn_decode_mma_takes(&a, hd)) return (int)cudaErrorNotSupported;
    if (r.qkv && ((a.page_table && (a.k_scale || a.v_scale)) || r.n_rot > 256 || r.n_rot > hd || (r.n_rot & 1) || (a.page_table ? r.n_rot && !r.freqs : !r.inv_freq))) return (int)cudaErrorNotSupported;
    if (a.page_table && (r.maps < 1 || r.maps > 2 || a.n_heads / a.n_kv_heads % r.maps || (r.maps > 1 && r.q_norm) || (r.no_append && r.q_norm))) return (int)cudaErrorInvalidValue;
    if (a.page_table && (!r.qkv || !r.neox || r.dim < 1 || r.maps * r.dim > hd || r.vdim < 1 || r.vdim > hd || r.n_rot > r.dim || a.max_pages < 1 || a.window < 0 || a.keep < 0 || r.v_off < 0 ||
                         (!r.no_append && r.v_off + a.n_kv_heads * r.vdim > r.ldq))) return (int)cudaErrorInvalidValue;
    return hd == 128 ? launch_d<128>(a, r, nb, pdl, st) : launch_d<64>(a, r, nb, pdl, st);
}

// Pipeline depth of the tensor-core decode kernel: 0 = chosen per launch (default), 2, 3 or 4 = forced (int8 caches: three at least).  Returns the previous setting.
B2_API int b2_attn_decode_stages(int n) {
    const int old = g_stages;
    if (n == 0 || (n >= 2 && n <= 4)) g_stages = n;
    return old;
}

// The depth of a launch for nb sequences.
B2_API int b2_attn_decode_depth(const AttnDecodeArgs* a, int nb) { return stages_for(*a, nb); }

int attn_decode_mma_launch(const AttnDecodeArgs& a, int nb, int hd, int pdl, cudaStream_t st) {
    const AttnRopeArgs none = {};
    return attn_decode_mma_rope_launch(a, none, nb, hd, pdl, st);
}
