// Causal prompt attention on the 5th-generation tensor cores (tcgen05 + tensor memory + TMA).
//
// One CTA owns 128 consecutive query rows of one query head of one sequence and walks the KV cache in
// tiles of 64 slots up to the last slot its rows may see:
//   S = Q K^T        tcgen05.mma, M = 128 rows, N = 64 slots, K = head dim; Q and the K tiles arrive by TMA
//                    (128-byte swizzle, no cluster broadcast) in the K-major layout the MMA reads; the scores of tile
//                    t + 1 are formed in a second buffer while those of tile t go through the soft-max;
//   soft-max         a row belongs to two threads (of the two warps that may read its lanes of tensor memory): both find
//                    its maximum, each forms the weights of 32 slots; they go to shared memory in the swizzled K-major
//                    layout (the A operand of the second product);
//   O += P V         tcgen05.mma, M = 128 rows, N = head dim, K = 64 slots.  V lies in the cache with the head dim
//                    contiguous, which is the MN-major form of this operand: its tiles arrive by TMA like K's.  O stays
//                    in tensor memory and is scaled by a warp only when the maximum of one of its rows grew.  (Weights
//                    that refer to an older maximum while it grows by less than 2^8 would save half of that, 1 % of a prompt of
//                    3001 rows, but the largest weight would no longer be exactly 1 in fp16: 15 % more error where the
//                    scores are peaked, 2-3 % elsewhere);
//   K and V tiles have two buffers each, so no step waits on global memory.
// The end: 1 / sum, the sigmoid output gate and the fp16 store.  Grouped-query heads share the K/V tiles through L2.
// Every mbarrier wait is bounded; on expiry the kernel records a status, frees its tensor memory and returns.
//
// Bound: the latencies of a step.  Measured: 3001 rows through 4 such layers of 16 heads of 256 and 4 others 16.9 -> 16.2 ms
// against a form with one phase after the other, V transposed by the threads and O scaled in registers every step.
//
// Replaces the reference's prefill attention kernels, which run 64-wide tiles on vector ALUs
// (reference: src/kernels/flash_attn_256_v3.hip:80,189, flash_attn_256_tuned.hip:200).
#include <cuda.h>
#include "kernels.cuh"
#include "tc_util.cuh"

#define AT_ROWS 128               // query rows per CTA (MMA M)
#define AT_KV 64                  // cache slots per tile
#define AT_THREADS 256

// byte offset of (row, 16-byte chunk c8 of its 128-byte line) in a K-major 128-byte-swizzled tile
__device__ __forceinline__ uint32_t at_sw(int row, int c8) { return (uint32_t)row * 128u + (uint32_t)((c8 ^ (row & 7)) << 4); }

// MN-major operand (128-byte swizzle): 64 elements of the contiguous dimension by 8 k in 1024 bytes, the next 64 elements
// `mn_stride` bytes on, the next 8 k 1024
__device__ __forceinline__ uint64_t make_desc_sw128_mn(uint32_t smem_addr, uint32_t mn_stride) {
    uint64_t d = make_desc_sw128(smem_addr);
    d &= ~((uint64_t)0x3FFF << 16);
    return d | (uint64_t)(mn_stride >> 4) << 16;
}
#define AT_IDESC_B_MN (1u << 16)              // B operand is MN-major
__device__ __forceinline__ void tc_st32f(uint32_t taddr, const float (&f)[32]) {
    uint32_t r[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(f[i]);
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
        :: "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
           "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
           "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
           "r"(r[31]), "r"(taddr) : "memory");
}

__device__ __forceinline__ void tc_ld32f(uint32_t taddr, float (&f)[32]) {
    uint32_t r[32];
    tc_ld32(taddr, r);
    tc_wait_ld();
#pragma unroll
    for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(r[i]);
}

template <int HD>
__global__ void __launch_bounds__(AT_THREADS, 1)
attn_prefill_tc_kernel(const AttnParams p, const __grid_constant__ CUtensorMap qmap,
                       const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, int row_base, int n_rows_seq, int* status) {
    constexpr int NB = HD / 64;                   // 64-wide blocks of the head dim (one swizzle line each)
    constexpr int OC = HD / 2;                    // output columns per thread
    extern __shared__ __align__(1024) unsigned char at_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)at_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sQ = smem;                                 // [NB][128 rows][128 B]
    constexpr int KB_BYTES = NB * AT_KV * 128;                // one K or V tile
    unsigned char* sK = sQ + (size_t)NB * AT_ROWS * 128;      // [2][NB][64 slots][128 B]
    unsigned char* sV = sK + (size_t)2 * KB_BYTES;            // [2][NB][64 slots][128 B]
    unsigned char* sP = sV + (size_t)2 * KB_BYTES;            // [128 rows][128 B]; at the end the row sums
    uint64_t* bars = (uint64_t*)(sP + (size_t)AT_ROWS * 128);
    uint64_t* k_full = bars;                                  // [2] K tile (and Q with the first)
    uint64_t* v_full = bars + 2;                              // [2] V tile
    uint64_t* s_done = bars + 4;                              // [2] scores of a tile
    uint64_t* o_done = bars + 6;                              // second product of a tile
    uint32_t* tmem_slot = (uint32_t*)(bars + 7);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int head = blockIdx.y, kvh = head / (p.nq / p.nkv);
    const int r0 = row_base + blockIdx.x * AT_ROWS;           // first row of this CTA in the launch
    const int r_end = row_base + n_rows_seq;
    constexpr int tmem_cols = HD == 256 ? 512 : 256;

    if (tid == 0) {
        for (int i = 0; i < 7; ++i) mbar_init(&bars[i], 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();                      // (not before this CTA has its tensor memory: csrc/gemm_tc.cu)
    pdl_wait();
    const uint32_t tmem_S = tmem_base, tmem_O = tmem_base + 2 * AT_KV;      // [2][64] columns of scores, then O

    // this thread's row: lane quarter (warp & 3) of tensor memory, row = 32 * (warp & 3) + lane
    const int lq = warp & 3, half = warp >> 2;
    const int row = lq * 32 + lane;
    const int gr = r0 + row;                                   // row in the launch
    const bool row_ok = gr < r_end;
    const RowMeta rm0 = p.rows[r0];
    const int seq = rm0.seq;
    const int my_ctx = row_ok ? p.rows[gr].ctx : 0;
    const int last = min(r0 + AT_ROWS, r_end) - 1;
    const int max_ctx = p.rows[last].ctx;                      // rows are in position order: the last sees the most
    const int n_tiles = (max_ctx + AT_KV - 1) / AT_KV;

    const uint32_t lanes = (uint32_t)(lq * 32) << 16;
    float m_ref = -INFINITY, l_run = 0.f;                      // (log2 domain; l_run: this thread's 32 slots of every tile)
    const float sc = p.scale * 1.44269504f;
    const uint32_t idesc_s = make_idesc_f16(AT_KV), idesc_o = make_idesc_f16(HD) | AT_IDESC_B_MN;
    const uint64_t dQ = make_desc_sw128(smem_u32(sQ)), dK = make_desc_sw128(smem_u32(sK));
    const uint64_t dP = make_desc_sw128(smem_u32(sP)), dV = make_desc_sw128_mn(smem_u32(sV), AT_KV * 128);
    bool ok = true;

    // tile t goes to buffer t & 1 (one lane of warp 0)
    auto issue = [&](int t, const CUtensorMap* map, unsigned char* buf, uint64_t* bar, bool with_q) {
        mbar_arrive_expect_tx(bar, (uint32_t)KB_BYTES + (with_q ? (uint32_t)NB * AT_ROWS * 128 : 0u));
        if (with_q)
            for (int b = 0; b < NB; ++b) tma_load_2d(sQ + (size_t)b * AT_ROWS * 128, &qmap, head * HD + b * 64, r0, bar);
        for (int b = 0; b < NB; ++b)
            tma_load_2d(buf + (size_t)(t & 1) * KB_BYTES + (size_t)b * AT_KV * 128, map, kvh * HD + b * 64, seq * p.max_seq + t * AT_KV, bar);
    };
    auto issue_k = [&](int t) { if (t < n_tiles && elect_one()) issue(t, &kmap, sK, &k_full[t & 1], t == 0); __syncwarp(); };
    auto issue_v = [&](int t) { if (t < n_tiles && elect_one()) issue(t, &vmap, sV, &v_full[t & 1], false); __syncwarp(); };
    // scores of tile t (warp 0); their buffer was last read in step t - 2
    auto scores = [&](int t) -> bool {
        if (t >= n_tiles) return true;
        if (!__all_sync(0xffffffffu, mbar_wait(&k_full[t & 1], (uint32_t)((t >> 1) & 1), abort_flag))) return false;
        tc_fence_after();
        if (elect_one()) {
            const uint64_t dKt = dK + (uint64_t)(((t & 1) * KB_BYTES) >> 4);
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int k16 = 0; k16 < 4; ++k16)
                    tc_mma_f16(tmem_S + (t & 1) * AT_KV, dQ + (uint64_t)((b * AT_ROWS * 128) >> 4) + 2 * k16,
                               dKt + (uint64_t)((b * AT_KV * 128) >> 4) + 2 * k16, idesc_s, (b | k16) ? 1u : 0u);
            tc_commit(&s_done[t & 1]);
        }
        __syncwarp();
        return true;
    };
    if (warp == 0) {
        issue_k(0); issue_v(0); issue_k(1); issue_v(1);
        ok = scores(0);
    }
    for (int tile = 0; tile < n_tiles; ++tile) {
        const int kv0 = tile * AT_KV;
        if (warp == 0 && ok) ok = scores(tile + 1);
        // (a thread whose wait gave up still walks to the next barrier, where the whole CTA decides to stop)
        ok = __all_sync(0xffffffffu, ok && mbar_wait(&s_done[tile & 1], (uint32_t)((tile >> 1) & 1), abort_flag));
        tc_fence_after();
        if (warp == 0 && ok) issue_k(tile + 2);                 // the scores of this tile have read its buffer
        float s[32], mx = -INFINITY;
        tc_ld32f(tmem_S + lanes + (tile & 1) * AT_KV + (half ^ 1) * 32, s);
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (kv0 + (half ^ 1) * 32 + i < my_ctx) mx = fmaxf(mx, s[i]);
        tc_ld32f(tmem_S + lanes + (tile & 1) * AT_KV + half * 32, s);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            s[i] = kv0 + half * 32 + i < my_ctx ? s[i] : -INFINITY;
            mx = fmaxf(mx, s[i]);
        }
        mx *= sc;
        const bool move = mx > m_ref;
        const float corr = move ? exp2f(m_ref - mx) : 1.f;
        if (move) m_ref = mx;
        const float ref = m_ref == -INFINITY ? 0.f : m_ref;
        uint32_t pk[16];
        float psum = 0.f;
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            const __half2 h2 = __floats2half2_rn(exp2f(s[i] * sc - ref), exp2f(s[i + 1] * sc - ref));
            // the sum uses the rounded values the second product sees
            psum += __low2float(h2) + __high2float(h2);
            pk[i >> 1] = *(const uint32_t*)&h2;
        }
        l_run = l_run * corr + psum;
        if (tile > 0) {
            ok = __all_sync(0xffffffffu, ok && mbar_wait(o_done, (uint32_t)((tile - 1) & 1), abort_flag));
            tc_fence_after();
            if (warp == 0 && ok) issue_v(tile + 1);             // the product of the tile before has read its buffer
            if (__any_sync(0xffffffffu, move)) {
#pragma unroll
                for (int c = 0; c < OC / 32; ++c) {
                    tc_ld32f(tmem_O + lanes + half * OC + c * 32, s);
#pragma unroll
                    for (int i = 0; i < 32; ++i) s[i] *= corr;
                    tc_st32f(tmem_O + lanes + half * OC + c * 32, s);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            *(uint4*)(sP + at_sw(row, half * 4 + q)) = make_uint4(pk[4 * q], pk[4 * q + 1], pk[4 * q + 2], pk[4 * q + 3]);
        if (kv0 + AT_KV > max_ctx) {
            // slots behind the last visible one hold what an earlier sequence left there: their weights are zero, but they
            // have to be finite
            ok = ok && mbar_wait(&v_full[tile & 1], (uint32_t)((tile >> 1) & 1), abort_flag);
            const int dead = max_ctx - kv0;                    // first such slot of the tile
            for (int i = tid; i < NB * (AT_KV - dead) * 8; i += AT_THREADS) {
                const int b = i / ((AT_KV - dead) * 8), r = i / 8 % (AT_KV - dead) + dead;
                *(uint4*)(sV + (size_t)(tile & 1) * KB_BYTES + (size_t)b * AT_KV * 128 + r * 128 + (i & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
            }
        }
        fence_proxy_async_smem();
        tc_fence_before();
        ok = __syncthreads_and(ok ? 1 : 0) != 0;
        if (!ok) break;
        // ---- O += P V
        if (warp == 0) {
            ok = __all_sync(0xffffffffu, mbar_wait(&v_full[tile & 1], (uint32_t)((tile >> 1) & 1), abort_flag));
            tc_fence_after();
            if (ok && elect_one()) {
                const uint64_t dVt = dV + (uint64_t)(((tile & 1) * KB_BYTES) >> 4);
#pragma unroll
                for (int k16 = 0; k16 < AT_KV / 16; ++k16)
                    tc_mma_f16(tmem_O, dP + 2 * k16, dVt + (uint64_t)(k16 * (2 * 1024 >> 4)), idesc_o, (tile | k16) ? 1u : 0u);
                tc_commit(o_done);
            }
            __syncwarp();
        }
    }
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    if (ok && n_tiles > 0) ok = mbar_wait(o_done, (uint32_t)((n_tiles - 1) & 1), abort_flag);
    tc_fence_after();
    float* sums = (float*)sP;                                  // [2][128]
    if (ok) sums[half * AT_ROWS + row] = l_run;
    __syncthreads();
    if (ok) {
        const float l = sums[row] + sums[AT_ROWS + row], inv = l > 0.f ? 1.f / l : 0.f;
        const size_t col0 = (size_t)head * HD + half * OC;
        __half* dst = p.out + (size_t)gr * p.ldo + col0;
        const __half* gq = p.gate_off >= 0 ? p.q + (size_t)gr * p.ldq + p.gate_off + col0 : nullptr;
        for (int c0 = 0; c0 < OC; c0 += 32) {
            float o[32];
            tc_ld32f(tmem_O + lanes + half * OC + c0, o);
#pragma unroll
            for (int c = 0; c < 32; c += 8) {
                if (!row_ok) break;
                uint4 gv = make_uint4(0u, 0u, 0u, 0u);
                if (gq) gv = *(const uint4*)(gq + c0 + c);
                const __half* gh = (const __half*)&gv;
                __half2 o2[4];
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    float a = o[c + e] * inv, b = o[c + e + 1] * inv;
                    if (gq) { a *= sigmoid_f(__half2float(gh[e])); b *= sigmoid_f(__half2float(gh[e + 1])); }
                    o2[e >> 1] = __floats2half2_rn(a, b);
                }
                *(uint4*)(dst + c0 + c) = *(const uint4*)o2;
            }
            __syncwarp();
        }
    }
    if (*abort_flag && tid == 0 && status) atomicExch(status, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(tmem_cols) : "memory");
}

static size_t at_smem(int hd) {
    const int nb = hd / 64;
    return 1024 + (size_t)nb * AT_ROWS * 128 + (size_t)4 * nb * AT_KV * 128 + (size_t)AT_ROWS * 128 + 96;
}

template <int HD>
static int launch_attn_prefill_tc(const AttnParams* p, const CUtensorMap& qmap, const CUtensorMap& kmap, const CUtensorMap& vmap, int row_base,
                                  int n_rows_seq, int* status, cudaStream_t s) {
    const size_t smem = at_smem(HD);
    static SmemOptIn opt;
    if (int e = opt.ensure(attn_prefill_tc_kernel<HD>, smem)) return e;
    dim3 grid((n_rows_seq + AT_ROWS - 1) / AT_ROWS, p->nq);
    return launch_pdl(attn_prefill_tc_kernel<HD>, grid, dim3(AT_THREADS), smem, s, *p, qmap, kmap, vmap, row_base, n_rows_seq, status);
}

// Rows [row_base, row_base + n_rows_seq) of the launch belong to one sequence, are in position order and carry
// no draft-tree masks (RowMeta.mask == 0); the cache already holds their own K/V rows.  n_slots: sequence slots
// of the cache (its first dimension).  status[0] is set to 1 when a bounded wait expired.
B2_API int b2_attn_prefill_tc(const AttnParams* p, int row_base, int n_rows_seq, int n_slots, int hd, int* status,
                              cudaStream_t s) {
    if (hd != 64 && hd != 128 && hd != 256) return cudaErrorInvalidValue;
    if (p->nq % p->nkv || n_rows_seq < 1 || (p->ldq & 7) || (p->ldo & 7) || ((uintptr_t)p->q & 15) || ((uintptr_t)p->out & 15) ||
        ((uintptr_t)p->kcache & 15) || ((uintptr_t)p->vcache & 15) || (p->gate_off >= 0 && (p->gate_off & 7)))
        return cudaErrorInvalidValue;
    EncodeTiledFn enc = get_encode();
    if (!enc) return cudaErrorNotSupported;
    CUtensorMap qmap, kmap, vmap;
    cuuint32_t estr[2] = {1, 1};
    {
        cuuint64_t dims[2] = {(cuuint64_t)p->nq * hd, (cuuint64_t)p->n_rows};
        cuuint64_t strides[1] = {(cuuint64_t)p->ldq * 2};
        cuuint32_t box[2] = {64, AT_ROWS};
        if (enc(&qmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)p->q, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    {
        cuuint64_t dims[2] = {(cuuint64_t)p->nkv * hd, (cuuint64_t)p->max_seq * n_slots};
        cuuint64_t strides[1] = {(cuuint64_t)p->nkv * hd * 2};
        cuuint32_t box[2] = {64, AT_KV};
        for (int v = 0; v < 2; ++v)
            if (enc(v ? &vmap : &kmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)(v ? p->vcache : p->kcache), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return cudaErrorInvalidValue;
    }
    if (hd == 256) return launch_attn_prefill_tc<256>(p, qmap, kmap, vmap, row_base, n_rows_seq, status, s);
    if (hd == 128) return launch_attn_prefill_tc<128>(p, qmap, kmap, vmap, row_base, n_rows_seq, status, s);
    return launch_attn_prefill_tc<64>(p, qmap, kmap, vmap, row_base, n_rows_seq, status, s);
}
