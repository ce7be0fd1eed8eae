// Tensor-core attention over the KV cache for many query rows: prompt processing, draft
// verification and batched decode.
//
// Rows of one sequence are taken 16 at a time; a CTA handles one such tile for one KV head and
// (optionally) one slice of the cache, with one warp per query head of the GQA group, so K and V
// are staged in shared memory once per group.  S = Q K^T and O += P V run on mma.sync m16n8k16
// (fp16 in, fp32 accumulate) with the online-softmax rescaling of flash attention; the visibility
// rule is the decode kernel's:  slot s is visible to a row iff  s < ctx  or  bit (s - ctx) of its
// mask is set, which covers causal prompts (ctx = position + 1) and draft trees (ctx = committed
// length, mask = the node's ancestors and itself).  The sigmoid output gate is applied in the
// epilogue.  This replaces the reference's prefill attention kernels and its tree-masked variant
// (reference: src/kernels/flash_attn_256.hip, src/kernels/flash_attn_256_v3.hip,
// src/kernels/flash_attn_tree.hip:74-193), which walk the keys with scalar dot products.
#include "kernels.cuh"

#define AR_ROWS 16               // query rows per tile
#define AR_KV 64                 // cache slots per block
#define AR_MAX_WARPS 8
#define AR_PAD 8                 // halfs of padding per shared-memory row (conflict-free ldmatrix)

__device__ __forceinline__ void ar_ldsm4(uint32_t (&r)[4], const __half* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ar_ldsm4_t(uint32_t (&r)[4], const __half* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ar_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_h2(float x, float y) {
    __half2 h = __floats2half2_rn(x, y);
    return *(uint32_t*)&h;
}

// Find the tile: sequences are consecutive row ranges (seq_rows), each cut into 16-row tiles.
__device__ __forceinline__ bool ar_find_tile(const int* seq_rows, int n_seqs, int tile, int& row0, int& nrows, int tile_rows = AR_ROWS) {
    for (int s = 0; s < n_seqs; ++s) {
        const int a = seq_rows[s], b = seq_rows[s + 1];
        const int nt = (b - a + tile_rows - 1) / tile_rows;
        if (tile < nt) { row0 = a + tile * tile_rows; nrows = min(tile_rows, b - row0); return true; }
        tile -= nt;
    }
    return false;
}

template <int HD>
__global__ void __launch_bounds__(AR_MAX_WARPS * 32, 1) attn_rows_kernel(const AttnParams p, const int* __restrict__ seq_rows,
                                                                        int n_seqs, int splits) {
    constexpr int LD = HD + AR_PAD;
    constexpr int NT_O = HD / 8;                 // 8-column tiles of the output
    pdl_launch_dependents();
    pdl_wait();
    int row0, nrows;
    if (!ar_find_tile(seq_rows, n_seqs, blockIdx.x, row0, nrows)) return;
    const int kvh = blockIdx.y, sp = blockIdx.z;
    const int G = p.nq / p.nkv;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x;
    const int g = lane >> 2, t = lane & 3;

    extern __shared__ __align__(16) unsigned char ar_smem[];
    __half* Qs = (__half*)ar_smem;                               // [G][16][LD]
    __half* Kb = Qs + (size_t)G * AR_ROWS * LD;                  // [2][64][LD]
    __half* Vb = Kb + 2 * AR_KV * LD;                            // [2][64][LD]

    // visibility of this thread's two rows (g and g + 8 of the tile)
    const RowMeta r_lo = p.rows[row0 + min(g, nrows - 1)], r_hi = p.rows[row0 + min(g + 8, nrows - 1)];
    const int ctx_lo = g < nrows ? r_lo.ctx : 0, ctx_hi = g + 8 < nrows ? r_hi.ctx : 0;
    const unsigned long long mk_lo = g < nrows ? r_lo.mask : 0ull, mk_hi = g + 8 < nrows ? r_hi.mask : 0ull;
    const int seq = r_lo.seq;
    // cache range the tile needs: the furthest visible slot over its rows (every thread computes the same value)
    int kv_end = 0;
    for (int r = 0; r < nrows; ++r) {
        const RowMeta rm = p.rows[row0 + r];
        const int extra = rm.mask ? 64 - __clzll((long long)rm.mask) : 0;
        kv_end = max(kv_end, min(rm.ctx + extra, p.max_seq));
    }
    const int n_blocks = (kv_end + AR_KV - 1) / AR_KV;
    const int per = (n_blocks + splits - 1) / splits;
    const int b_begin = sp * per, b_end = min(n_blocks, b_begin + per);

    // ---- stage Q (all heads of the group) and the first K/V block
    const size_t kv_base = ((size_t)seq * p.max_seq) * p.nkv * HD + (size_t)kvh * HD;
    const size_t kv_stride = (size_t)p.nkv * HD;
    constexpr int PPR = HD / 8;                                  // 16-byte pieces per row
    for (int idx = tid; idx < G * AR_ROWS * PPR; idx += nthr) {
        const int pc = idx % PPR, r = (idx / PPR) % AR_ROWS, h = idx / (PPR * AR_ROWS);
        __half* dst = Qs + ((size_t)h * AR_ROWS + r) * LD + pc * 8;
        if (r < nrows) cp_async16(dst, p.q + (size_t)(row0 + r) * p.ldq + (size_t)(kvh * G + h) * HD + pc * 8);
        else *(uint4*)dst = make_uint4(0u, 0u, 0u, 0u);
    }
    auto stage_kv = [&](int blk, int buf) {
        for (int idx = tid; idx < AR_KV * PPR; idx += nthr) {
            const int pc = idx % PPR, r = idx / PPR;
            const int slot = blk * AR_KV + r;
            __half* kd = Kb + ((size_t)buf * AR_KV + r) * LD + pc * 8;
            __half* vd = Vb + ((size_t)buf * AR_KV + r) * LD + pc * 8;
            if (slot < kv_end) {
                cp_async16(kd, p.kcache + kv_base + (size_t)slot * kv_stride + pc * 8);
                cp_async16(vd, p.vcache + kv_base + (size_t)slot * kv_stride + pc * 8);
            } else {
                *(uint4*)kd = make_uint4(0u, 0u, 0u, 0u);
                *(uint4*)vd = make_uint4(0u, 0u, 0u, 0u);
            }
        }
    };
    if (b_begin < b_end) stage_kv(b_begin, 0);
    cp_async_commit();

    float o[NT_O][4];
#pragma unroll
    for (int n = 0; n < NT_O; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    float m_lo = -INFINITY, m_hi = -INFINITY, l_lo = 0.f, l_hi = 0.f;
    const bool active = warp < G;
    const __half* qw = Qs + (size_t)warp * AR_ROWS * LD;
    const int a_row = (lane & 7) + ((lane >> 3) & 1) * 8, a_col = (lane >> 4) * 8;      // A operand (row-major) addressing
    const int b_row = (lane & 7) + (lane >> 4) * 8, b_col = ((lane >> 3) & 1) * 8;      // B operand from [n][k] storage
    const float sc = p.scale * 1.44269504f;                      // scores are kept in the log2 domain

    for (int blk = b_begin; blk < b_end; ++blk) {
        const int buf = (blk - b_begin) & 1;
        cp_async_wait<0>();
        __syncthreads();                                         // block `blk` landed; everyone left block blk-1
        if (blk + 1 < b_end) stage_kv(blk + 1, buf ^ 1);
        cp_async_commit();
        if (!active) continue;
        const __half* Kt = Kb + (size_t)buf * AR_KV * LD;
        const __half* Vt = Vb + (size_t)buf * AR_KV * LD;
        // ---- S = Q K^T  (16 x 64)
        float s[AR_KV / 8][4];
#pragma unroll
        for (int n = 0; n < AR_KV / 8; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll 2
        for (int k0 = 0; k0 < HD; k0 += 16) {
            uint32_t a[4];
            ar_ldsm4(a, qw + a_row * LD + k0 + a_col);
#pragma unroll
            for (int np = 0; np < AR_KV / 16; ++np) {
                uint32_t b[4];
                ar_ldsm4(b, Kt + (np * 16 + b_row) * LD + k0 + b_col);
                ar_mma(s[2 * np], a, b[0], b[1]);
                ar_mma(s[2 * np + 1], a, b[2], b[3]);
            }
        }
        // ---- mask, online softmax
        const int s_base = blk * AR_KV;
        float mx_lo = -INFINITY, mx_hi = -INFINITY;
#pragma unroll
        for (int n = 0; n < AR_KV / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int slot = s_base + 8 * n + 2 * t + (e & 1);
                const bool hi = e >= 2;
                const int ctx = hi ? ctx_hi : ctx_lo;
                const unsigned long long mk = hi ? mk_hi : mk_lo;
                const int d = slot - ctx;
                const bool vis = d < 0 || (d < 64 && ((mk >> d) & 1ull));
                const float v = vis ? s[n][e] * sc : -INFINITY;
                s[n][e] = v;
                if (hi) mx_hi = fmaxf(mx_hi, v); else mx_lo = fmaxf(mx_lo, v);
            }
        mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 1)); mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 2));
        mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 1)); mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 2));
        const float mn_lo = fmaxf(m_lo, mx_lo), mn_hi = fmaxf(m_hi, mx_hi);
        const float ref_lo = mn_lo == -INFINITY ? 0.f : mn_lo, ref_hi = mn_hi == -INFINITY ? 0.f : mn_hi;
        const float cor_lo = exp2f(m_lo - ref_lo), cor_hi = exp2f(m_hi - ref_hi);      // exp2(-inf) = 0 for the first block
        m_lo = mn_lo; m_hi = mn_hi;
        float rs_lo = 0.f, rs_hi = 0.f;
        uint32_t pa[AR_KV / 16][4];
#pragma unroll
        for (int n = 0; n < AR_KV / 8; ++n) {
            const float p0 = exp2f(s[n][0] - ref_lo), p1 = exp2f(s[n][1] - ref_lo);
            const float p2 = exp2f(s[n][2] - ref_hi), p3 = exp2f(s[n][3] - ref_hi);
            rs_lo += p0 + p1; rs_hi += p2 + p3;
            // two adjacent 8-column score tiles form the A fragment of one 16-slot step of P V
            pa[n >> 1][(n & 1) * 2 + 0] = pack_h2(p0, p1);
            pa[n >> 1][(n & 1) * 2 + 1] = pack_h2(p2, p3);
        }
        l_lo = l_lo * cor_lo + rs_lo; l_hi = l_hi * cor_hi + rs_hi;
#pragma unroll
        for (int n = 0; n < NT_O; ++n) { o[n][0] *= cor_lo; o[n][1] *= cor_lo; o[n][2] *= cor_hi; o[n][3] *= cor_hi; }
        // ---- O += P V
#pragma unroll
        for (int k16 = 0; k16 < AR_KV / 16; ++k16) {
#pragma unroll
            for (int np = 0; np < NT_O / 2; ++np) {
                uint32_t b[4];
                ar_ldsm4_t(b, Vt + (k16 * 16 + a_row) * LD + np * 16 + a_col);
                ar_mma(o[2 * np], pa[k16], b[0], b[1]);
                ar_mma(o[2 * np + 1], pa[k16], b[2], b[3]);
            }
        }
    }
    cp_async_wait<0>();
    if (!active) return;
    // row sums live in the four lanes of a row quad
    l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 1); l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 2);
    l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 1); l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 2);
    const int head = kvh * G + warp;
    if (splits == 1) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = g + 8 * half;
            if (r >= nrows) continue;
            const float inv = 1.f / (half ? l_hi : l_lo);
            const size_t row = (size_t)(row0 + r);
#pragma unroll
            for (int n = 0; n < NT_O; ++n) {
                const int col = 8 * n + 2 * t;
                float v0 = o[n][2 * half] * inv, v1 = o[n][2 * half + 1] * inv;
                if (p.gate_off >= 0) {
                    const __half2 gt = *(const __half2*)(p.q + row * p.ldq + p.gate_off + (size_t)head * HD + col);
                    v0 *= sigmoid_f(__low2float(gt)); v1 *= sigmoid_f(__high2float(gt));
                }
                *(__half2*)(p.out + row * p.ldo + (size_t)head * HD + col) = __floats2half2_rn(v0, v1);
            }
        }
    } else {
        // partial result of this slice: unnormalised O, running maximum (log2 domain) and sum
        // scratch: [row][head][split][HD + 2]
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = g + 8 * half;
            if (r >= nrows) continue;
            float* dst = p.scratch + (((size_t)(row0 + r) * p.nq + head) * splits + sp) * (HD + 2);
#pragma unroll
            for (int n = 0; n < NT_O; ++n)
                *(float2*)(dst + 8 * n + 2 * t) = make_float2(o[n][2 * half], o[n][2 * half + 1]);
            if (t == 0) { dst[HD] = half ? m_hi : m_lo; dst[HD + 1] = half ? l_hi : l_lo; }
        }
    }
}

// Few rows per sequence (drafts, batched decode): the group's heads are packed into the rows of the MMA tiles (unit
// u = row * G + head, 16 MT units per CTA), so that a tile is not mostly padding, and the warps divide the slots of a
// block instead of the heads: warp (m, q) scores its 16 units against slots 16 q .. of every block and keeps its own
// running maximum, sum and output; the four parts of a tile meet once, in shared memory, at the end.  K and V leave
// shared memory MT times instead of G times, Q stays in registers, and nothing is multiplied for rows that do not exist.
// Bound: the cache (265 MB for 16 sequences of 4051 slots, 4 heads of 256).  Measured there, 5 rows x 6 heads: 71 us a
// layer against 166 with a warp per head.
template <int HD, int MT>
__global__ void __launch_bounds__(MT * 128, 1) attn_rows_packed_kernel(const AttnParams p, const int* __restrict__ seq_rows,
                                                                      int n_seqs, int splits, int tile_rows) {
    constexpr int LD = HD + AR_PAD, NT_O = HD / 8, THREADS = MT * 128, PPR = HD / 8;
    pdl_launch_dependents();
    pdl_wait();
    int row0, nrows;
    if (!ar_find_tile(seq_rows, n_seqs, blockIdx.x, row0, nrows, tile_rows)) return;
    const int kvh = blockIdx.y, sp = blockIdx.z, G = p.nq / p.nkv, units = nrows * G;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, mt = warp >> 2, part = warp & 3;
    const int g = lane >> 2, t = lane & 3;

    extern __shared__ __align__(16) unsigned char ar_smem[];
    __half* Qs = (__half*)ar_smem;                               // [16 MT][LD]
    __half* Kb = Qs + MT * AR_ROWS * LD;                         // [2][64][LD]
    __half* Vb = Kb + 2 * AR_KV * LD;                            // [2][64][LD]

    // visibility of this thread's two units
    const int u_lo = mt * 16 + g, u_hi = u_lo + 8;
    const RowMeta r_lo = p.rows[row0 + min(u_lo / G, nrows - 1)], r_hi = p.rows[row0 + min(u_hi / G, nrows - 1)];
    const int ctx_lo = u_lo < units ? r_lo.ctx : 0, ctx_hi = u_hi < units ? r_hi.ctx : 0;
    const unsigned long long mk_lo = u_lo < units ? r_lo.mask : 0ull, mk_hi = u_hi < units ? r_hi.mask : 0ull;
    const int seq = r_lo.seq;
    int kv_end = 0;
    for (int r = 0; r < nrows; ++r) {
        const RowMeta rm = p.rows[row0 + r];
        const int extra = rm.mask ? 64 - __clzll((long long)rm.mask) : 0;
        kv_end = max(kv_end, min(rm.ctx + extra, p.max_seq));
    }
    const int n_blocks = (kv_end + AR_KV - 1) / AR_KV;
    const int per = (n_blocks + splits - 1) / splits;
    const int b_begin = sp * per, b_end = min(n_blocks, b_begin + per);

    const size_t kv_base = ((size_t)seq * p.max_seq) * p.nkv * HD + (size_t)kvh * HD;
    const size_t kv_stride = (size_t)p.nkv * HD;
    for (int idx = tid; idx < MT * AR_ROWS * PPR; idx += THREADS) {
        const int pc = idx % PPR, u = idx / PPR;
        __half* dst = Qs + (size_t)u * LD + pc * 8;
        if (u < units) cp_async16(dst, p.q + (size_t)(row0 + u / G) * p.ldq + (size_t)(kvh * G + u % G) * HD + pc * 8);
        else *(uint4*)dst = make_uint4(0u, 0u, 0u, 0u);
    }
    auto stage_kv = [&](int blk, int buf) {
        for (int idx = tid; idx < AR_KV * PPR; idx += THREADS) {
            const int pc = idx % PPR, r = idx / PPR, slot = blk * AR_KV + r;
            __half* kd = Kb + ((size_t)buf * AR_KV + r) * LD + pc * 8;
            __half* vd = Vb + ((size_t)buf * AR_KV + r) * LD + pc * 8;
            if (slot < kv_end) {
                cp_async16(kd, p.kcache + kv_base + (size_t)slot * kv_stride + pc * 8);
                cp_async16(vd, p.vcache + kv_base + (size_t)slot * kv_stride + pc * 8);
            } else {
                *(uint4*)kd = make_uint4(0u, 0u, 0u, 0u);
                *(uint4*)vd = make_uint4(0u, 0u, 0u, 0u);
            }
        }
    };
    cp_async_commit();
    if (b_begin < b_end) stage_kv(b_begin, 0);
    cp_async_commit();
    const int a_row = (lane & 7) + ((lane >> 3) & 1) * 8, a_col = (lane >> 4) * 8;      // A operand (row-major) addressing
    const int b_row = (lane & 7) + (lane >> 4) * 8, b_col = ((lane >> 3) & 1) * 8;      // B operand from [n][k] storage
    cp_async_wait<1>();
    __syncthreads();
    uint32_t qf[HD / 16][4];
#pragma unroll
    for (int k = 0; k < HD / 16; ++k) ar_ldsm4(qf[k], Qs + (mt * 16 + a_row) * LD + k * 16 + a_col);

    float o[NT_O][4];
#pragma unroll
    for (int n = 0; n < NT_O; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    float m_lo = -INFINITY, m_hi = -INFINITY, l_lo = 0.f, l_hi = 0.f;
    const float sc = p.scale * 1.44269504f;                      // scores are kept in the log2 domain

    for (int blk = b_begin; blk < b_end; ++blk) {
        const int buf = (blk - b_begin) & 1;
        cp_async_wait<0>();
        __syncthreads();                                         // block `blk` landed; everyone left block blk-1
        if (blk + 1 < b_end) stage_kv(blk + 1, buf ^ 1);
        cp_async_commit();
        const __half* Kt = Kb + ((size_t)buf * AR_KV + part * 16) * LD;
        const __half* Vt = Vb + ((size_t)buf * AR_KV + part * 16) * LD;
        // ---- S = Q K^T  (16 x 16), even and odd k steps in chains of their own
        float s[2][4], s2[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[n][e] = s2[n][e] = 0.f;
#pragma unroll
        for (int k = 0; k < HD / 16; k += 2) {
            uint32_t b[4], c[4];
            ar_ldsm4(b, Kt + b_row * LD + k * 16 + b_col);
            ar_ldsm4(c, Kt + b_row * LD + (k + 1) * 16 + b_col);
            ar_mma(s[0], qf[k], b[0], b[1]);
            ar_mma(s[1], qf[k], b[2], b[3]);
            ar_mma(s2[0], qf[k + 1], c[0], c[1]);
            ar_mma(s2[1], qf[k + 1], c[2], c[3]);
        }
        // ---- mask, online softmax
        const int s_base = blk * AR_KV + part * 16;
        float mx_lo = -INFINITY, mx_hi = -INFINITY;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int d = s_base + 8 * n + 2 * t + (e & 1) - (e >= 2 ? ctx_hi : ctx_lo);
                const bool vis = d < 0 || (d < 64 && (((e >= 2 ? mk_hi : mk_lo) >> d) & 1ull));
                const float v = vis ? (s[n][e] + s2[n][e]) * sc : -INFINITY;
                s[n][e] = v;
                if (e >= 2) mx_hi = fmaxf(mx_hi, v); else mx_lo = fmaxf(mx_lo, v);
            }
        mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 1)); mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 2));
        mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 1)); mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 2));
        const float mn_lo = fmaxf(m_lo, mx_lo), mn_hi = fmaxf(m_hi, mx_hi);
        const float ref_lo = mn_lo == -INFINITY ? 0.f : mn_lo, ref_hi = mn_hi == -INFINITY ? 0.f : mn_hi;
        // (the output is scaled only when some maximum of the warp moved)
        if (__any_sync(0xffffffffu, mn_lo != m_lo || mn_hi != m_hi)) {
            const float cor_lo = exp2f(m_lo - ref_lo), cor_hi = exp2f(m_hi - ref_hi);      // exp2(-inf) = 0 for the first block
            l_lo *= cor_lo; l_hi *= cor_hi;
#pragma unroll
            for (int n = 0; n < NT_O; ++n) { o[n][0] *= cor_lo; o[n][1] *= cor_lo; o[n][2] *= cor_hi; o[n][3] *= cor_hi; }
        }
        m_lo = mn_lo; m_hi = mn_hi;
        uint32_t pa[4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const float p0 = exp2f(s[n][0] - ref_lo), p1 = exp2f(s[n][1] - ref_lo);
            const float p2 = exp2f(s[n][2] - ref_hi), p3 = exp2f(s[n][3] - ref_hi);
            l_lo += p0 + p1; l_hi += p2 + p3;
            pa[n * 2 + 0] = pack_h2(p0, p1);
            pa[n * 2 + 1] = pack_h2(p2, p3);
        }
        // ---- O += P V
#pragma unroll
        for (int np = 0; np < NT_O / 2; ++np) {
            uint32_t b[4];
            ar_ldsm4_t(b, Vt + a_row * LD + np * 16 + a_col);
            ar_mma(o[2 * np], pa, b[0], b[1]);
            ar_mma(o[2 * np + 1], pa, b[2], b[3]);
        }
    }
    cp_async_wait<0>();
    l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 1); l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 2);
    l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 1); l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 2);
    __syncthreads();                                             // every warp left the last block: its memory holds the parts
    constexpr int OLD = HD + 8;                                  // (rows 8 banks apart: the 8-byte stores of a half warp meet none twice)
    float* Os = (float*)ar_smem;                                 // [4 MT][16][OLD], column HD: maximum, HD + 1: sum
    {
        float* a = Os + ((size_t)warp * 16 + g) * OLD;
        float* b = a + 8 * OLD;
#pragma unroll
        for (int n = 0; n < NT_O; ++n) {
            *(float2*)(a + 8 * n + 2 * t) = make_float2(o[n][0], o[n][1]);
            *(float2*)(b + 8 * n + 2 * t) = make_float2(o[n][2], o[n][3]);
        }
        if (t == 0) { a[HD] = m_lo; a[HD + 1] = l_lo; b[HD] = m_hi; b[HD + 1] = l_hi; }
    }
    __syncthreads();
    for (int idx = tid; idx < units * (HD / 2); idx += THREADS) {
        const int u = idx / (HD / 2), col = idx % (HD / 2) * 2, row = row0 + u / G, head = kvh * G + u % G;
        const float* a = Os + ((size_t)(u >> 4) * 64 + (u & 15)) * OLD;
        float m = -INFINITY;
#pragma unroll
        for (int q = 0; q < 4; ++q) m = fmaxf(m, a[q * 16 * OLD + HD]);
        const float ref = m == -INFINITY ? 0.f : m;
        float l = 0.f, v0 = 0.f, v1 = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float w = exp2f(a[q * 16 * OLD + HD] - ref);
            const float2 v = *(const float2*)(a + q * 16 * OLD + col);
            l = fmaf(a[q * 16 * OLD + HD + 1], w, l);
            v0 = fmaf(v.x, w, v0); v1 = fmaf(v.y, w, v1);
        }
        if (splits == 1) {
            const float inv = 1.f / l;
            v0 *= inv; v1 *= inv;
            if (p.gate_off >= 0) {
                const __half2 gt = *(const __half2*)(p.q + (size_t)row * p.ldq + p.gate_off + (size_t)head * HD + col);
                v0 *= sigmoid_f(__low2float(gt)); v1 *= sigmoid_f(__high2float(gt));
            }
            *(__half2*)(p.out + (size_t)row * p.ldo + (size_t)head * HD + col) = __floats2half2_rn(v0, v1);
        } else {
            float* dst = p.scratch + (((size_t)row * p.nq + head) * splits + sp) * (HD + 2);
            *(float2*)(dst + col) = make_float2(v0, v1);
            if (col == 0) { dst[HD] = m; dst[HD + 1] = l; }
        }
    }
}

// Merge the slices of split attention: one warp per (row, head).
#define MERGE 4                  // slices whose parts are requested at once
template <int HD>
__global__ void __launch_bounds__(128) attn_rows_merge_kernel(const AttnParams p, int splits) {
    pdl_launch_dependents();
    pdl_wait();
    const int item = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (item >= p.n_rows * p.nq) return;
    const int row = item / p.nq, head = item % p.nq;
    const float* src = p.scratch + (size_t)item * splits * (HD + 2);
    constexpr int EPL = HD / 32;
    // Everything the merge needs of the first MERGE slices is on its way before anything is used, the gates too: read between the
    // stores of the output they were a trip to L2 for each element (24 rows, three slices, 24 launches: 2.86 -> 2.76 ms; 80 rows, two
    // slices, 16 launches: 11.01 -> 10.89).  What bounds it: one trip to L2 and the launch
    const __half* gate = p.q + (size_t)row * p.ldq + max(p.gate_off, 0) + (size_t)head * HD + lane * EPL;
    __half* out = p.out + (size_t)row * p.ldo + (size_t)head * HD + lane * EPL;
    const bool vec = ((p.ldq | max(p.gate_off, 0) | p.ldo) & (EPL - 1)) == 0 && (((uintptr_t)p.q | (uintptr_t)p.out) & (2 * EPL - 1)) == 0;
    uint32_t gw[EPL / 2], ow[EPL / 2];
#pragma unroll
    for (int e = 0; e < EPL / 2; ++e) gw[e] = 0u;
    if (p.gate_off >= 0) {
        if (vec) {
            if constexpr (EPL == 8) { const uint4 g = *(const uint4*)gate; gw[0] = g.x; gw[1] = g.y; gw[2] = g.z; gw[3] = g.w; }
            else
#pragma unroll
                for (int e = 0; e < EPL / 2; ++e) gw[e] = ((const uint32_t*)gate)[e];
        } else
#pragma unroll
            for (int e = 0; e < EPL / 2; ++e) { const __half2 h = __halves2half2(gate[2 * e], gate[2 * e + 1]); gw[e] = *(const uint32_t*)&h; }
    }
    float2 v[MERGE][EPL / 2], ml[MERGE];                     // (slices are HD + 2 floats apart: 8-byte loads)
    auto load = [&](int s0) {
#pragma unroll
        for (int u = 0; u < MERGE; ++u) {
            const float2* ps = (const float2*)(src + (size_t)min(s0 + u, splits - 1) * (HD + 2));
            ml[u] = ps[HD / 2];
#pragma unroll
            for (int e = 0; e < EPL / 2; ++e) v[u][e] = ps[lane * (EPL / 2) + e];
        }
    };
    load(0);
    float m = -INFINITY;
    for (int s = MERGE; s < splits; ++s) m = fmaxf(m, src[(size_t)s * (HD + 2) + HD]);
#pragma unroll
    for (int u = 0; u < MERGE; ++u) if (u < splits) m = fmaxf(m, ml[u].x);
    if (m == -INFINITY) m = 0.f;
    float acc[EPL], l = 0.f;
#pragma unroll
    for (int e = 0; e < EPL; ++e) acc[e] = 0.f;
    for (int s0 = 0; s0 < splits; s0 += MERGE) {
        if (s0) load(s0);
#pragma unroll
        for (int u = 0; u < MERGE; ++u) {
            if (s0 + u >= splits) break;
            const float w = exp2f(ml[u].x - m);
            l += ml[u].y * w;
#pragma unroll
            for (int e = 0; e < EPL / 2; ++e) { acc[2 * e] += v[u][e].x * w; acc[2 * e + 1] += v[u][e].y * w; }
        }
    }
    const float inv = 1.f / l;
#pragma unroll
    for (int e = 0; e < EPL / 2; ++e) {
        const float2 g = __half22float2(*(const __half2*)&gw[e]);
        float a = acc[2 * e] * inv, b = acc[2 * e + 1] * inv;
        if (p.gate_off >= 0) { a *= sigmoid_f(g.x); b *= sigmoid_f(g.y); }
        const __half2 h = __floats2half2_rn(a, b);
        ow[e] = *(const uint32_t*)&h;
        if (!vec) { out[2 * e] = __low2half(h); out[2 * e + 1] = __high2half(h); }
    }
    if (vec) {
        if constexpr (EPL == 8) *(uint4*)out = make_uint4(ow[0], ow[1], ow[2], ow[3]);
        else
#pragma unroll
            for (int e = 0; e < EPL / 2; ++e) ((uint32_t*)out)[e] = ow[e];
    }
}

template <int HD, int MT>
static int launch_packed(const AttnParams* p, const int* seq_rows, int n_seqs, int splits, int tile_rows, cudaStream_t s) {
    size_t smem = ((size_t)MT * AR_ROWS + 4 * AR_KV) * (HD + AR_PAD) * sizeof(__half);
    const size_t parts = (size_t)MT * 64 * (HD + 8) * sizeof(float);
    if (smem < parts) smem = parts;
    static SmemOptIn optin;
    if (cudaError_t e = optin.ensure(attn_rows_packed_kernel<HD, MT>, smem)) return e;
    const int tiles = (p->n_rows + tile_rows - 1) / tile_rows + n_seqs;       // upper bound; surplus CTAs exit at once
    return launch_pdl(attn_rows_packed_kernel<HD, MT>, dim3(tiles, p->nkv, splits), dim3(MT * 128), smem, s, *p, seq_rows, n_seqs, splits, tile_rows);
}

template <int HD>
static int launch_rows(const AttnParams* p, const int* seq_rows, int n_seqs, int splits, cudaStream_t s) {
    const int G = p->nq / p->nkv;
    const size_t smem = ((size_t)G * AR_ROWS + 4 * AR_KV) * (HD + AR_PAD) * sizeof(__half);
    static SmemOptIn optin;
    {
        cudaError_t e = optin.ensure(attn_rows_kernel<HD>, smem);
        if (e != cudaSuccess) return e;
    }
    // heads packed into the tiles while the rows of a sequence (on average) fit two tiles of them: a second CTA of the
    // same sequence would read the cache again, and from there on a warp per head wastes less than that
    const int units = (p->n_rows + n_seqs - 1) / n_seqs * G;
    cudaError_t e;
    if (units <= 16) e = (cudaError_t)launch_packed<HD, 1>(p, seq_rows, n_seqs, splits, 16 / G, s);
    else if (units <= 32) e = (cudaError_t)launch_packed<HD, 2>(p, seq_rows, n_seqs, splits, 32 / G, s);
    else {
        const int tiles = (p->n_rows + AR_ROWS - 1) / AR_ROWS + n_seqs;       // upper bound; surplus CTAs exit at once
        dim3 grid(tiles, p->nkv, splits);
        e = launch_pdl(attn_rows_kernel<HD>, grid, dim3(G * 32), smem, s, *p, seq_rows, n_seqs, splits);
    }
    if (e != cudaSuccess || splits == 1) return e;
    return launch_pdl(attn_rows_merge_kernel<HD>, dim3((p->n_rows * p->nq + 3) / 4), dim3(128), 0, s, *p, splits);
}

// p->splits: cache slices per tile (1 = none; needs scratch of n_rows * nq * splits * (hd + 2) floats).
B2_API int b2_attn_rows(const AttnParams* p, const int* seq_rows, int n_seqs, int hd, cudaStream_t s) {
    const int G = p->nkv > 0 ? p->nq / p->nkv : 0;
    if (G < 1 || G > AR_MAX_WARPS || p->nq % p->nkv || n_seqs < 1 || p->splits < 1) return cudaErrorInvalidValue;
    if (hd == 256) return launch_rows<256>(p, seq_rows, n_seqs, p->splits, s);
    if (hd == 64) return launch_rows<64>(p, seq_rows, n_seqs, p->splits, s);
    return cudaErrorInvalidValue;
}
