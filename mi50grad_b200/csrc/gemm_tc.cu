// Dense-weight GEMM of many rows on the 5th-generation tensor cores:
//   C[t][n] = sum_k X[t][k] * W[n][k],  X and W fp16 or both bf16, fp32 accumulation in tensor memory.
//
// Replaces the reference's fp16 prefill GEMMs (reference: src/kernels/gemm_fp16_prefill.hip:47,
// gemm_fp16_prefill_silu_dual.hip:62), which run 64x64x16 tiles on vector ALUs.  (INT4 weights: csrc/gemm_int4.cu.)
//
// One CTA computes a [128 outputs x T tokens] tile (T <= 512, all of tensor memory), or [256 x T] with T <= 256:
//   * the WEIGHT tile is the MMA's A operand (M = 128 outputs), the activations are the B
//     operand (N = tokens, any multiple of 16 up to 256 per instruction), so a batch of 16..80 rows costs no padding;
//   * warp 16 brings both tiles with TMA (cp.async.bulk.tensor, 128-byte swizzle, no cluster broadcast) onto the
//     stage's mbarrier;
//   * warp 17 issues tcgen05.mma (cta_group::1, kind::f16) on shared-memory descriptors and
//     releases stages with tcgen05.commit; both single-lane roles keep their warp converged and
//     elect a lane only around the tcgen05 / TMA instructions;
//   * warps 0-15 then read the accumulators back with tcgen05.ld and run the epilogue.
// Every mbarrier wait is bounded; on expiry the kernel records a status, skips the rest of
// its work, releases its tensor memory and returns.
#include <cuda.h>
#include "kernels.cuh"
#include "gemm_tc.cuh"
#include "tc_util.cuh"
#include "gemm_epilogue.cuh"

#define TC_EPI_WARPS 16
#define TC_THREADS ((TC_EPI_WARPS + 2) * 32)
#define TC_BK 64                 // k per stage (128 bytes of fp16: one swizzle row)
#define TC_BM 128                // outputs per CTA (MMA M)
#define TC_A_BYTES (TC_BM * TC_BK * 2)

// PAIR: the kernel of CTA pairs is an instantiation of its own: a kernel that contains cta_group::2 instructions
// cannot be launched without a cluster (the plain launch is refused with "invalid cluster size").
template <bool PAIR>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_dense_tc_kernel(const GemmTcParams p, const __grid_constant__ CUtensorMap xmap,
                    const __grid_constant__ CUtensorMap wmap) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // the dynamic window is only guaranteed 16-byte aligned: align to the 1024-byte swizzle atom by hand
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    // (the broadcast and the votes below tell the compiler that roles and loop exits are warp-uniform: descriptors
    // and stage counters then stay in uniform registers, which takes about 70 cycles off a k-block)
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int S = p.stages;
    const int t0 = blockIdx.y * p.t_tile;
    const int Tp = (min(p.t_tile, p.T - t0) + 15) & ~15;          // token columns of this CTA
    // (a CTA pair multiplies whole 256-token operand tiles: rows beyond T are zero-filled by the loads)
    const int Tm = PAIR ? (Tp + 255) & ~255 : Tp;
    const int box = p.box_rows, boxes = (Tp + box - 1) / box;     // token rows per TMA load
    // (CTA pairs: a CTA stages only its half of the token rows)
    const int b_stage_bytes = ((p.t_tile + 63) / 64) * 64 * 128 / (PAIR ? 2 : 1);
    // MH = 2: the CTA owns 256 outputs as two M = 128 accumulators that share every activation tile (half the
    // activation bytes per FLOP)
    // pair: two CTAs of a cluster (adjacent output tiles) run their MMAs as one cta_group::2 instruction stream,
    // M = 256 over the two SMs: each CTA loads its own 128 weight rows and only ITS half of every
    // 256-token operand tile, so the shared-memory traffic of the token operand per SM halves
    constexpr bool pair = PAIR;
    uint32_t crank = 0u;
    if constexpr (PAIR) crank = cluster_ctarank();
    const int MH = p.m_halves == 2 ? 2 : 1;
    const int a_bytes = MH * TC_A_BYTES;
    unsigned char* sA = smem;
    unsigned char* sB = smem + (size_t)S * a_bytes;
    uint64_t* bars = (uint64_t*)(sB + (size_t)S * b_stage_bytes);
    uint64_t* full = bars;              // [S] 1 arrival with the TMA transaction bytes
    uint64_t* empty = bars + S;         // [S] 1 arrival (tcgen05.commit)
    uint64_t* acc_full = bars + 2 * S;  // 1 arrival
    uint64_t* peer_full = bars + 2 * S + 1;   // [S] pair mode, leader CTA: the peer's operands of the stage are in place
    uint32_t* tmem_slot = (uint32_t*)(bars + 3 * S + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    int tmem_cols = 32;
    while (tmem_cols < Tm) tmem_cols <<= 1;
    if (MH == 2) tmem_cols = 512;                  // accumulator h at column 256 h (Tp <= 256)

    if (tid == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_full, 1);
        for (int s = 0; s < S; ++s) mbar_init(&peer_full[s], 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (PAIR) cluster_sync_all();       // both CTAs' barriers exist before anyone signals the other
    if (warp == TC_EPI_WARPS) {
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                         :: "r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                         :: "r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Programmatic launch: the next kernel may start once every CTA of this one has its tensor memory (a CTA of the next
    // that took it first would wait for this kernel while this one waited for it).  This one starts likewise while the kernel
    // before it ends: barriers and tensor memory are ready when the activations are.
    pdl_launch_dependents();
    if (!p.w_older) pdl_wait();
    // split-K: this CTA's k-blocks are [kb_lo, kb_lo + KB) of the p.KB blocks of the matrix
    const int per_kb = (p.KB + (int)gridDim.z - 1) / (int)gridDim.z;
    const int kb_lo = (int)blockIdx.z * per_kb;
    const int KB = max(0, min(p.KB, kb_lo + per_kb) - kb_lo);

    // Every role walks the stages with running counters (stage index, phase bit, addresses).  The
    // loops of the single-thread roles are chains of dependent instructions, so each instruction
    // taken out of them shortens the time per k-block directly.
    if (warp < TC_EPI_WARPS) {
        // ================= epilogue =================
        // (one lane polls, the other epilogue warps sleep at a hardware barrier: hundreds of polling threads slow the TMA and
        // MMA warps down)
        if (warp == 0) {
            if (lane == 0) mbar_wait(acc_full, 0, abort_flag);
            __syncwarp();
        }
        asm volatile("bar.sync 1, %0;" :: "n"(TC_EPI_WARPS * 32) : "memory");
        pdl_wait();
        tc_fence_after();
        if (!*abort_flag) {
            const int lg = warp & 3;               // tensor-memory lane group this warp may read
            const size_t plane = (size_t)blockIdx.z * (size_t)p.plane_stride;     // (split-K of TC_EPI_STORE_F32)
            // (the operands' stages are free: their products are done)
            unsigned char* stage = smem + warp * TC_EPI_STAGE;
            const int Tn = min(p.t_tile, p.T - t0), chunks = (Tn + TC_EPI_COLS - 1) / TC_EPI_COLS;
            for (int c = warp >> 2; c < MH * chunks; c += TC_EPI_WARPS / 4) {
                const int hc = c >= chunks ? 1 : 0, c0 = (c - hc * chunks) * TC_EPI_COLS;
                uint32_t r[TC_EPI_COLS];
                tc_ld16(tmem_base + ((uint32_t)(lg * 32) << 16) + (uint32_t)(hc * 256 + c0), r);
                tc_wait_ld();
                tc_epilogue(p, r, lane, blockIdx.x * (TC_BM * MH) + hc * TC_BM + lg * 32, t0 + c0, Tn - c0, plane, gridDim.z > 1, stage);
            }
        }
    } else if (warp == TC_EPI_WARPS) {
        // ================= operand producer (TMA) =================
        {
            // pair mode: of every 256-token operand tile this CTA loads rows [128 crank, 128 crank + 128)
            const uint32_t tx = (pair ? (uint32_t)(Tm / 2) * 128u : (uint32_t)(boxes * box) * 128u) + (uint32_t)a_bytes;
            const int row_w = blockIdx.x * (TC_BM * MH);
            pdl_wait();
            int st = 0;
            uint32_t ph = 0;
            unsigned char* a = sA;
            unsigned char* b = sB;
            for (int kb = 0, kx = kb_lo * TC_BK; kb < KB; ++kb, kx += TC_BK) {
                if (!__all_sync(0xffffffffu, mbar_wait(&empty[st], ph ^ 1, abort_flag, 64))) break;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&full[st], tx);
                    for (int hc = 0; hc < MH; ++hc) tma_load_2d(a + hc * TC_A_BYTES, &wmap, kx, row_w + hc * TC_BM, &full[st]);
                    if (pair) {
                        for (int j = 0; j < Tm / 256; ++j)
                            for (int bx = 0; bx < 2; ++bx)
                                tma_load_2d(b + j * (128 * 128) + bx * (64 * 128), &xmap, kx, t0 + j * 256 + (int)crank * 128 + bx * 64, &full[st]);
                    } else {
                        for (int bx = 0; bx < boxes; ++bx)
                            tma_load_2d(b + bx * (box * 128), &xmap, kx, t0 + bx * box, &full[st]);
                    }
                }
                __syncwarp();
                a += a_bytes; b += b_stage_bytes;
                if (++st == S) { st = 0; ph ^= 1; a = sA; b = sB; }
            }
        }
    } else {
        // ================= MMA issuer =================
        {
            const int n1 = min(Tp, 256), n2 = Tp - n1;
            const uint32_t fmt = p.bf16 ? TC_IDESC_BF16 : 0u;
            const uint32_t idesc1 = make_idesc_f16(n1) | fmt, idesc2 = make_idesc_f16(n2 > 0 ? n2 : 16) | fmt;
            // descriptors differ between stages and k16 steps only in the start-address field (16-byte units)
            const uint64_t ad0 = make_desc_sw128(smem_u32(sA)), bd0 = make_desc_sw128(smem_u32(sB));
            const uint64_t a_step = (uint64_t)(a_bytes >> 4), b_step = (uint64_t)(b_stage_bytes >> 4), b_half = (256 * 128) >> 4;
            const uint64_t a_half = TC_A_BYTES >> 4;
            uint64_t ad = ad0, bd = bd0;
            int st = 0;
            uint32_t ph = 0;
            bool ok = true;
            const uint32_t idesc_pair = make_idesc_f16_m256(256) | fmt;
            const uint64_t b_pair_half = (128 * 128) >> 4;
            for (int kb = 0; kb < KB; ++kb) {
                ok = __all_sync(0xffffffffu, mbar_wait(&full[st], ph, abort_flag, 64));
                if (!ok) break;
                if constexpr (PAIR) {
                    if (crank != 0) {
                        // peer CTA: its operands of the stage are in place: tell the leader, which issues for both
                        if (elect_one()) mbar_arrive_remote(&peer_full[st], 0);
                        __syncwarp();
                        if (++st == S) { st = 0; ph ^= 1; }
                        continue;
                    }
                    ok = mbar_wait_cluster(&peer_full[st], ph, abort_flag);
                    if (!ok) break;
                }
                tc_fence_after();
                if constexpr (PAIR) {
                    if (elect_one()) {
#pragma unroll
                        for (int k16 = 0; k16 < TC_BK / 16; ++k16)
                            for (int j = 0; j < Tm / 256; ++j)
                                tc_mma_f16_pair(tmem_base + 256 * j, ad + 2 * k16, bd + j * b_pair_half + 2 * k16, idesc_pair, (kb | k16) ? 1u : 0u);
                        tc_commit_pair(&empty[st]);
                    }
                    __syncwarp();
                    ad += a_step; bd += b_step;
                    if (++st == S) { st = 0; ph ^= 1; ad = ad0; bd = bd0; }
                    continue;
                }
                if (elect_one()) {
#pragma unroll
                    for (int k16 = 0; k16 < TC_BK / 16; ++k16) {
                        tc_mma_f16(tmem_base, ad + 2 * k16, bd + 2 * k16, idesc1, (kb | k16) ? 1u : 0u);
                        if (MH == 2) tc_mma_f16(tmem_base + 256, ad + a_half + 2 * k16, bd + 2 * k16, idesc1, (kb | k16) ? 1u : 0u);
                        else if (n2 > 0) tc_mma_f16(tmem_base + 256, ad + 2 * k16, bd + b_half + 2 * k16, idesc2, (kb | k16) ? 1u : 0u);
                    }
                    tc_commit(&empty[st]);      // stage reusable once these MMAs have read it
                }
                __syncwarp();
                ad += a_step; bd += b_step;
                if (++st == S) { st = 0; ph ^= 1; ad = ad0; bd = bd0; }
            }
            if constexpr (PAIR) { if (ok && crank == 0 && elect_one()) tc_commit_pair(acc_full); }
            else { if (ok && elect_one()) tc_commit(acc_full); }
            __syncwarp();
        }
    }
    if (*abort_flag && tid == 0 && p.status) atomicExch(p.status, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if constexpr (PAIR) cluster_sync_all();       // neither CTA frees tensor memory (or leaves) while the pair's MMAs or
                                                  // the other CTA's signals may still touch it
    if (warp == TC_EPI_WARPS) {
        if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static size_t dense_smem(int t_tile, int stages, int m_halves) {
    size_t b = (size_t)((t_tile + 63) / 64) * 64 * 128;
    return 1024 + (size_t)stages * ((size_t)(m_halves == 2 ? 2 : 1) * TC_A_BYTES + b) + (3 * stages + 1) * 8 + 16 + 16;
}

// x: [T][ldx] fp16 activations (ldx multiple of 8, base 16-byte aligned).
static int launch_tc(const GemmTcParams* p, const void* w, int ldw, int n_rows_w, const void* x, int ldx,
                     cudaStream_t stream) {
    if (p->T < 1 || p->t_tile < 16 || p->t_tile > 512 || (p->t_tile & 15) || (ldx & 7) || ((uintptr_t)x & 15))
        return cudaErrorInvalidValue;
    EncodeTiledFn enc = get_encode();
    if (!enc) return cudaErrorNotSupported;
    CUtensorMap map;
    cuuint64_t dims[2] = {(cuuint64_t)p->K, (cuuint64_t)p->T};
    cuuint64_t strides[1] = {(cuuint64_t)ldx * 2};
    // (as few loads per k-block as a box of at most 256 rows allows; a CTA's stage holds t_tile rounded up to 64)
    const int box_rows = p->cta_pair ? 64 : (p->t_tile <= 256 ? (p->t_tile + 63) / 64 * 64 : (p->t_tile % 256 ? 64 : 256));
    cuuint32_t box[2] = {TC_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    const CUtensorMapDataType dtype = p->bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUresult r = enc(&map, dtype, 2, (void*)x, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    CUtensorMap wmap;
    if ((ldw & 7) || ((uintptr_t)w & 15)) return cudaErrorInvalidValue;
    cuuint64_t wd[2] = {(cuuint64_t)p->K, (cuuint64_t)n_rows_w};
    cuuint64_t ws[1] = {(cuuint64_t)ldw * 2};
    cuuint32_t wb[2] = {TC_BK, TC_BM};
    r = enc(&wmap, dtype, 2, (void*)w, wd, ws, wb, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    GemmTcParams q = *p;
    q.box_rows = box_rows;
    // 256-output tiles: only with at most 256 tokens per CTA (two accumulators of 256 columns; rows behind the last are
    // zero-filled and not stored)
    if (q.m_halves != 2 || q.t_tile > 256) q.m_halves = 1;
    dim3 grid((q.NTL * 16 + TC_BM * q.m_halves - 1) / (TC_BM * q.m_halves), (q.T + q.t_tile - 1) / q.t_tile, 1);
    // CTA pairs: 256-token operand tiles, an even number of 128-output CTAs (a surplus tile is made up: its rows are
    // zero-filled and not stored)
    if (q.cta_pair && q.m_halves == 1) grid.x += grid.x & 1;
    if (q.cta_pair && (q.m_halves != 1 || (grid.x & 1) || (q.t_tile != 256 && q.t_tile != 512))) q.cta_pair = 0;
    const size_t per_stage = (size_t)q.m_halves * TC_A_BYTES + (size_t)((q.t_tile + 63) / 64) * 64 * 128 / (q.cta_pair ? 2 : 1);
    // as many stages as shared memory holds; deep pipelines matter most for few tokens, where a stage is consumed quickly
    int stages = (int)((227 * 1024 - 1024 - 256) / per_stage);
    q.stages = stages > 8 ? 8 : (stages < 2 ? 2 : stages);
    const size_t smem = dense_smem(q.cta_pair ? q.t_tile / 2 : q.t_tile, q.stages, q.m_halves);
    static SmemOptIn optin;
    {
        cudaError_t e = optin.ensure(gemm_dense_tc_kernel<false>, smem);
        if (e != cudaSuccess) return e;
    }
    const bool planes = q.epi == TC_EPI_STORE_F32 && q.plane_stride > 0 && q.softcap <= 0.f;
    int ks = ((q.epi == TC_EPI_RESID_F32 || planes) && q.k_splits > 1) ? q.k_splits : 1;
    if (ks > q.KB) ks = q.KB;
    if (ks > 1) { const int per = (q.KB + ks - 1) / ks; ks = (q.KB + per - 1) / per; }     // no empty split
    grid.z = ks;
    if (q.cta_pair) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid; cfg.blockDim = dim3(TC_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;
        static SmemOptIn optin_pair;
        if (cudaError_t e = optin_pair.ensure(gemm_dense_tc_kernel<true>, smem)) return e;
        return cudaLaunchKernelEx(&cfg, gemm_dense_tc_kernel<true>, q, map, wmap);
    }
    return launch_pdl(gemm_dense_tc_kernel<false>, grid, dim3(TC_THREADS), smem, stream, q, map, wmap);
}
// fp16 or bf16 (p->bf16) weights w[N][ldw] (row = output feature).  p->K, T, t_tile, n_valid (= N), ldo, epi, out, status are
// used; the INT4 fields are ignored.
B2_API int b2_gemm_f16_tc(const GemmTcParams* p, const void* w, int ldw, const void* x, int ldx, cudaStream_t stream) {
    if (!w || p->n_valid < 1) return cudaErrorInvalidValue;
    GemmTcParams q = *p;
    q.KB = (q.K + TC_BK - 1) / TC_BK;        // a ragged last block is zero-filled by both TMA loads
    const int n_rows_w = q.epi == TC_EPI_SILU_PAIR ? 2 * q.n_valid : q.n_valid;      // (gate / up rows interleaved by 8)
    q.NTL = (n_rows_w + TC_BM - 1) / TC_BM * (TC_BM / 16);
    q.qfrag = nullptr; q.szfrag = nullptr;
    return launch_tc(&q, w, ldw, n_rows_w, x, ldx, stream);
}
B2_API int b2_sizeof_gemm_tc_params() { return (int)sizeof(GemmTcParams); }
