// Many-row INT4 GEMM on the 5th-generation tensor cores:
//   C[t][n] = sum_k X[t][k] * W[k][n],  X fp16 activations, W INT4 (group-wise scale/zero), fp32 accumulation in tensor memory.
//
// Replaces the reference's prefill GEMM family (reference: src/kernels/gemm_int4_prefill_hip.hip:27,
// gemm_int4_prefill_v2.hip:41, src/asm/gemm_*.s), which runs 64x64x16 tiles on vector ALUs.
//
// The WEIGHT tile is the MMA's A operand (M = 128 outputs) and comes from TENSOR MEMORY; the activations are the B operand
// (N = tokens, any multiple of 16) in shared memory.  A CTA, one on an SM, has [128 MH outputs x t_tile tokens x a range of K].
//   * warps 0-15 dequantise.  A lane's packed weights of a 16 x 64 tile are one 16-byte load (fragment order of the decode
//     GEMV), held two steps ahead in registers; expanded to fp16 ((q - zero) * scale, the 0x6400 trick) they are in the
//     order of tcgen05.st.16x128b, so they go from registers into tensor memory as they are.
//   * warp 16 brings the activation tiles with TMA (128-byte swizzle, no cluster broadcast) and asks for the weights
//     some k-blocks ahead in L2;
//   * warp 17 (and 18: one for each accumulator) issues tcgen05.mma (A in tensor memory) and releases slots and stages
//     with tcgen05.commit.
//   * warps 0-15 then read the accumulators back and store them.
// Tensor memory (512 columns): MH accumulators of t_tile columns and four slots of weights, two for each group of eight
// dequantising warps; a slot has [128 outputs x 64 KS k].
//
// Why tensor memory: with the dequantised tile in shared memory its stores waited for the operand reads of the MMAs, which go
// first: four stmatrix and a proxy fence of 16 warps took 600-1270 cycles beside them, tcgen05.st of the same tile takes
// 65-105.  It also takes the A operand off the shared-memory port (n = 16: 75 instead of 157 cycles a k-block).
// (CTAs that walk over several tiles, with the first weights of a tile before the epilogue of the one before, or over equal
// shares of all tiles' k-blocks, were no faster than as many CTAs and splits over K: what they have to keep in mind costs
// the dequantising warps 2 us in 20 with few tokens.)
// What bounds it (block_us in csrc/driver.cu has the measured k-block times): many tokens, the tensor pipe; few tokens, the latency
// from a weight's load to its products, no unit: with 80 tokens (5120 -> 34816) 54 % of the issue slots are busy, the tensor pipe 45 % of
// the time, 30 % of the memory bandwidth is used, and a warp waits for loads 3.3 of the 8.9 cycles between two instructions.
// Every mbarrier wait is bounded; on expiry the kernel records a status, skips the rest of its work, releases its tensor
// memory and returns.
#include <cuda.h>
#include "kernels.cuh"
#include "gemm_tc.cuh"
#include "tc_util.cuh"
#include "gemm_epilogue.cuh"

#define TS_PRODUCERS 16           // dequantising warps (also the epilogue warps), two groups of 8
#define TS_BK 64                  // k of a k-block (128 bytes of fp16: one swizzle row)
#define TS_BM 128
#define TS_SLOTS 4
#define TS_MAX_STAGES 16
#define TS_STAGE_SMEM (192 * 1024)
// k-blocks that the weights are requested ahead into L2, in front of the two steps that are held in registers.  256 outputs, 16 tokens,
// 37888 x 5120: 28.6 us; 8 ahead 29.8, 24 ahead 31.2; nothing 27.5, but then 128 outputs take 4 % longer
#define TS_AHEAD 4

__device__ __forceinline__ uint32_t ts_nib_lo(uint32_t w) {
    uint32_t r;
    asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xea;" : "=r"(r) : "r"(w));
    return r;
}
__device__ __forceinline__ uint32_t ts_nib_hi(uint32_t w) {
    uint32_t r;
    asm("lop3.b32 %0, %1, 0x00f000f0, 0x64006400, 0xea;" : "=r"(r) : "r"(w));
    return r;
}
__device__ __forceinline__ uint4 ts_load_w(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void ts_prefetch_l2(const void* p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ts_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        :: "r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// 16 lanes x 32 columns: register 2 i + j of lane (g, t) = lane >> 2, lane & 3 is row g + 8 j, k = 8 i + 2 t and 8 i + 2 t + 1
__device__ __forceinline__ void ts_store(uint32_t a, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        :: "r"(a), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
           "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void ts_wait_store() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 k of a 16-row tile (words w0, w1 of a lane) -> r[0..7]
__device__ __forceinline__ void ts_dequant(uint32_t w0, uint32_t w1, uint2 sz, uint32_t* r) {
    const __half2 sixteenth = __float2half2_rn(0.0625f), k1024 = __float2half2_rn(1024.f), k64 = __float2half2_rn(64.f);
    const __half2 s2 = *(const __half2*)&sz.x, z2 = *(const __half2*)&sz.y;
    const __half2 s_lo = __half2half2(__low2half(s2)), s_hi = __half2half2(__high2half(s2));
    const __half2 z_lo = __half2half2(__low2half(z2)), z_hi = __half2half2(__high2half(z2));
    const __half2 cl_lo = __hadd2(k1024, z_lo), cl_hi = __hadd2(k1024, z_hi);                  // 1024 + zero
    const __half2 ch_lo = __hneg2(__hadd2(k64, z_lo)), ch_hi = __hneg2(__hadd2(k64, z_hi));   // -(64 + zero)
    auto lo = [&](uint32_t x, __half2 c, __half2 sc) {
        uint32_t q = ts_nib_lo(x);
        const __half2 v = __hmul2(__hsub2(*(__half2*)&q, c), sc);
        return *(const uint32_t*)&v;
    };
    auto hi = [&](uint32_t x, __half2 c, __half2 sc) {
        uint32_t q = ts_nib_hi(x);
        const __half2 v = __hmul2(__hfma2(*(__half2*)&q, sixteenth, c), sc);
        return *(const uint32_t*)&v;
    };
    r[0] = lo(w0, cl_lo, s_lo); r[1] = lo(w0 >> 8, cl_hi, s_hi);
    r[2] = lo(w1, cl_lo, s_lo); r[3] = lo(w1 >> 8, cl_hi, s_hi);
    r[4] = hi(w0, ch_lo, s_lo); r[5] = hi(w0 >> 8, ch_hi, s_hi);
    r[6] = hi(w1, ch_lo, s_lo); r[7] = hi(w1 >> 8, ch_hi, s_hi);
}

// MH: accumulators of 128 outputs.  KS: k-blocks per slot and stage: two, since a slot's waits, commits and
// instructions around them cost an MMA warp as much as the products of few tokens, or one where the accumulators leave
// room for no more.  UNI: a pair of k-blocks is a group of 128, with one scale per output; else every 32 k look theirs up.
template <int MH, int KS, bool UNI>
__global__ void __launch_bounds__((TS_PRODUCERS + 1 + MH) * 32, 1)
gemm_int4_ts_kernel(const GemmTcParams p, const __grid_constant__ CUtensorMap xmap, const int n_mt, const int n_tt, const int per_kb) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* sB = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);      // [S][KS][t_tile rows of 128 bytes]
    // (the broadcast and the votes below tell the compiler that roles and loop exits are warp-uniform)
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    unsigned char* sE = sB + (size_t)p.stages * (KS * p.t_tile * 128);                          // [16] staging of the epilogue
    const int S = p.stages, box_bytes = p.t_tile * 128, stage_bytes = KS * box_bytes;
    uint64_t* b_full = (uint64_t*)(sE + TS_PRODUCERS * TC_EPI_STAGE);   // [S] the TMA bytes
    uint64_t* b_empty = b_full + S;                 // [S] a commit of every MMA warp
    uint64_t* a_full = b_empty + S;                 // [4] one arrival per warp of the group
    uint64_t* a_empty = a_full + TS_SLOTS;          // [4] a commit
    uint64_t* acc_full = a_empty + TS_SLOTS;        // a commit of every MMA warp
    uint32_t* tmem_slot = (uint32_t*)(acc_full + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int acc_cols = (p.t_tile + 31) & ~31;     // columns of an accumulator

    if (tid == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], MH); }
        for (int s = 0; s < TS_SLOTS; ++s) { mbar_init(&a_full[s], TS_PRODUCERS / 2); mbar_init(&a_empty[s], 1); }
        mbar_init(acc_full, MH);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == TS_PRODUCERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + 512 - TS_SLOTS * 32 * KS;
    // Programmatic launch: the next kernel may start once every CTA of this one has its tensor memory (a CTA of the next
    // that took it first would wait for this kernel while this one waited for it).  This one starts likewise while the kernel
    // before it ends: only the TMA warp and the epilogue wait for it, the weights, which nothing in a step writes, are read at once.
    pdl_launch_dependents();
    if (!p.w_older) pdl_wait();

    // output tile mt, token tile tt, K range z; the token tiles of an output tile run side by side and share its weights in L2
    const int z = (int)blockIdx.x / (n_mt * n_tt), tile = (int)blockIdx.x - z * (n_mt * n_tt);
    const int mt = tile / n_tt, tt = tile - mt * n_tt;
    const int kb0 = z * per_kb, kbs = min(p.KB - kb0, per_kb);

    if (warp < TS_PRODUCERS) {
        // ================= dequantising warps, then epilogue =================
        // A step is a pair of k-blocks of one 16-row tile.  MH = 1: the two groups take alternate pairs; MH = 2: group h
        // takes every pair of accumulator h.  A warp reaches the tensor-memory lanes 32 (warp & 3) .. + 31, so its row tile
        // in the 128 outputs is 2 (warp & 3) + (bit 2 of the warp).
        const int grp = warp >> 3, rt = 2 * (warp & 3) + ((warp >> 2) & 1), g = lane >> 2;
        constexpr int NSZ = UNI ? 1 : 4;
        uint4 wq[2][2] = {};
        uint2 sz[2][NSZ] = {};
        const int first = MH == 2 ? 0 : grp, stride = MH == 2 ? 1 : 2, steps = (kbs + 1) >> 1;     // steps of this group
        const int wt = (mt * MH + (MH == 2 ? grp : 0)) * 2 + (rt >> 2);
        const uint4* l_q = p.qfrag + (((size_t)wt * p.KB + kb0 + 2 * first) * 4 + (rt & 3)) * 32 + lane;
        const uint2* l_s = p.szfrag + ((size_t)wt * p.G * 4 + (rt & 3)) * 8 + g;
        if (UNI) l_s += (size_t)(((p.off32 + 2 * kb0) >> 2) + first) * 32;
        int l_step = first;
        if (first >= steps) { l_q = p.qfrag + (((size_t)wt * p.KB + kb0) * 4 + (rt & 3)) * 32 + lane; if (UNI) l_s -= first * 32; }
        // (buffers 0 and 1 take the steps in turn)
        // A step behind the last reads the last again, a half one its first block twice: no branch stands between the loads.
        auto load = [&](int b) __attribute__((always_inline)) {
            wq[b][0] = ts_load_w(l_q);
            wq[b][1] = ts_load_w(l_q + (2 * l_step + 1 < kbs ? 128 : 0));
            if (UNI) sz[b][0] = __ldg(l_s);
            else {
                const int c = p.off32 + 2 * (kb0 + 2 * l_step);
#pragma unroll
                for (int j = 0; j < NSZ; ++j) sz[b][j] = __ldg(l_s + (size_t)min((c + j) >> p.gshift, p.G - 1) * 32);
            }
            l_step += stride;
            if (l_step < steps) {
                l_q += stride * 256;
                if (UNI) l_s += stride * 32;
            }
        };
        load(0);
        load(1);
        const uint32_t a_lane = tmem_a + ((uint32_t)(rt * 16) << 16) + (uint32_t)(grp * 2 * 32 * KS);
        bool ok = true;
        uint32_t q = 0;                            // slots that this group has filled: it has two, in turn
        // (with a whole step a slot the buffers alternate just as the slots do)
        auto slot = [&](int b) __attribute__((always_inline)) { return KS == 2 ? b : (int)(q & 1); };
        auto wait_slot = [&](int b) __attribute__((always_inline)) {
            uint64_t* bar = &a_empty[grp * 2 + slot(b)];
            const uint32_t parity = ((q >> 1) & 1) ^ 1;
            if (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
                int o = 1;
                if (lane == 0) o = mbar_wait(bar, parity, abort_flag) ? 1 : 0;   // (one lane polls)
                ok = __shfl_sync(0xffffffffu, o, 0) != 0;
            }
            tc_fence_after();
        };
        auto filled = [&](int b) __attribute__((always_inline)) {
            ts_wait_store();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[grp * 2 + slot(b)]);
            ++q;
        };
        auto step = [&](int b, int i) __attribute__((always_inline)) {
            const bool two = 2 * i + 1 < kbs;
            uint32_t r[16];
            ts_dequant(wq[b][0].x, wq[b][0].y, sz[b][0], r);
            ts_dequant(wq[b][0].z, wq[b][0].w, sz[b][UNI ? 0 : 1], r + 8);
            wait_slot(b);
            if (!ok) return;
            ts_store(a_lane + slot(b) * 32 * KS, r);
            if (KS == 1) filled(b);
            if (two) {
                ts_dequant(wq[b][1].x, wq[b][1].y, sz[b][UNI ? 0 : 2], r);
                ts_dequant(wq[b][1].z, wq[b][1].w, sz[b][UNI ? 0 : 3], r + 8);
                if (KS == 1) { wait_slot(b); if (!ok) return; }
                ts_store(a_lane + slot(b) * 32 * KS + (KS - 1) * 32, r);
            }
            load(b);
            if (KS == 2 || two) filled(b);
        };
        for (int s = first; s < steps; s += 2 * stride) {
            step(0, s);
            if (!ok) break;
            if (s + stride < steps) step(1, s + stride);
            if (!ok) break;
        }
        // ---- epilogue (one lane polls, the other warps sleep at a hardware barrier)
        if (warp == 0) {
            if (lane == 0 && ok) mbar_wait(acc_full, 0, abort_flag);
            __syncwarp();
        }
        asm volatile("bar.sync 1, %0;" :: "n"(TS_PRODUCERS * 32) : "memory");
        pdl_wait();
        ok = ok && !*abort_flag;
        tc_fence_after();
        if (ok) {
            const int lg = warp & 3, t0 = tt * p.t_tile, Tn = min(p.t_tile, p.T - t0);
            const size_t plane = (size_t)z * (size_t)p.plane_stride;     // (split-K of TC_EPI_STORE_F32)
            const int chunks = (Tn + TC_EPI_COLS - 1) / TC_EPI_COLS;
            for (int c = warp >> 2; c < MH * chunks; c += TS_PRODUCERS / 4) {
                const int hc = MH == 2 && c >= chunks ? 1 : 0, c0 = (c - hc * chunks) * TC_EPI_COLS;
                uint32_t r[TC_EPI_COLS];
                tc_ld16(tmem_base + ((uint32_t)(lg * 32) << 16) + (uint32_t)(hc * acc_cols + c0), r);
                tc_wait_ld();
                tc_epilogue(p, r, lane, (mt * MH + hc) * TS_BM + lg * 32, t0 + c0, Tn - c0, plane, per_kb < p.KB, sE + warp * TC_EPI_STAGE);
            }
        }
    } else if (warp == TS_PRODUCERS) {
        // ================= activation producer (TMA) =================
        int st = 0;
        uint32_t ph = 0;
        unsigned char* b = sB;
        const unsigned char* w0 = (const unsigned char*)(p.qfrag + ((size_t)mt * (2 * MH) * p.KB + kb0) * 128);
        // (2 KB of weights a k-block and 64 outputs, k-blocks side by side)
        auto ahead = [&](int kb, int n) {
            n = min(n, kbs - kb);
            if (n > 0) for (int j = 0; j < 2 * MH; ++j) ts_prefetch_l2(w0 + ((size_t)j * p.KB + kb) * 2048, (uint32_t)n * 2048u);
        };
        if (elect_one()) ahead(0, TS_AHEAD);
        __syncwarp();
        pdl_wait();
        for (int kb = 0, kx = kb0 * TS_BK; kb < kbs; kb += KS, kx += KS * TS_BK) {
            if (!__all_sync(0xffffffffu, mbar_wait(&b_empty[st], ph ^ 1, abort_flag))) break;
            if (elect_one()) {
                const bool two = KS == 2 && kb + 1 < kbs;
                mbar_arrive_expect_tx(&b_full[st], (uint32_t)(two ? 2 * box_bytes : box_bytes));
                tma_load_2d(b, &xmap, kx, tt * p.t_tile, &b_full[st]);
                if (two) tma_load_2d(b + box_bytes, &xmap, kx + TS_BK, tt * p.t_tile, &b_full[st]);
                if ((kb & 3) == 0) ahead(kb + TS_AHEAD, 4);
            }
            __syncwarp();
            b += stage_bytes;
            if (++st == S) { st = 0; ph ^= 1; b = sB; }
        }
    } else {
        // ================= MMA issuers: warp 17 + h for accumulator h =================
        // descriptors differ between stages and k16 steps only in the start-address field (16-byte units)
        const int h = MH == 2 ? warp - TS_PRODUCERS - 1 : 0;
        const uint64_t bd0 = make_desc_sw128(smem_u32(sB)), b_step = (uint64_t)(stage_bytes >> 4), b_box = (uint64_t)(box_bytes >> 4);
        const uint32_t acc = tmem_base + h * acc_cols, idesc = make_idesc_f16((min(p.t_tile, p.T - tt * p.t_tile) + 15) & ~15);
        uint64_t bd = bd0;
        int st = 0;
        uint32_t ph = 0;
        uint32_t q[2] = {0, 0};                    // slots of the group taken; MH = 2: only that of group h counts
        uint32_t odd = 0;                          // MH = 1: pairs of k-blocks come from the groups in turn
        bool ok = true;
        for (int kb = 0; kb < kbs; kb += KS) {
            const uint32_t grp = MH == 2 ? (uint32_t)h : odd;
            const uint32_t n = MH == 2 || !odd ? q[0] : q[1];
            const uint32_t sl = grp * 2 + (n & 1);
            // (both barriers are asked before either answer is needed)
            const bool r0 = mbar_try_wait(&b_full[st], ph), r1 = mbar_try_wait(&a_full[sl], (n >> 1) & 1);
            if (!__all_sync(0xffffffffu, r0 && r1)) {
                ok = __all_sync(0xffffffffu, mbar_wait(&b_full[st], ph, abort_flag) && mbar_wait(&a_full[sl], (n >> 1) & 1, abort_flag));
                if (!ok) break;
            }
            tc_fence_after();
            const uint32_t a = tmem_a + sl * (32 * KS);
            if (elect_one()) {
#pragma unroll
                for (int k16 = 0; k16 < TS_BK / 16; ++k16) ts_mma(acc, a + 8 * k16, bd + 2 * k16, idesc, (kb | k16) ? 1u : 0u);
                if (KS == 2 && kb + 1 < kbs) {
#pragma unroll
                    for (int k16 = 0; k16 < TS_BK / 16; ++k16) ts_mma(acc, a + 32 + 8 * k16, bd + b_box + 2 * k16, idesc, 1u);
                }
                tc_commit(&a_empty[sl]);
                tc_commit(&b_empty[st]);
            }
            __syncwarp();
            if (MH == 2 || !odd) ++q[0]; else ++q[1];
            if (MH == 1) odd ^= 1;
            bd += b_step;
            if (++st == S) { st = 0; ph ^= 1; bd = bd0; }
        }
        if (ok && elect_one()) tc_commit(acc_full);
        __syncwarp();
    }
    if (*abort_flag && tid == 0 && p.status) atomicExch(p.status, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == TS_PRODUCERS)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(512) : "memory");
}

// x: [T][ldx] fp16 activations (ldx multiple of 8, base 16-byte aligned).  t_tile, m_halves and k_splits are the wanted
// shape; a CTA takes at most 256 tokens with 128 outputs and 192 with 256 (their accumulators leave room for the weights).
B2_API int b2_gemm_int4_tc(const GemmTcParams* p, const void* x, int ldx, cudaStream_t stream) {
    if (p->bf16) return cudaErrorInvalidValue;             // INT4 weights are dequantised to fp16
    if (p->T < 1 || p->t_tile < 16 || p->t_tile > 512 || (p->t_tile & 15) || (ldx & 7) || ((uintptr_t)x & 15))
        return cudaErrorInvalidValue;
    EncodeTiledFn enc = get_encode();
    if (!enc) return cudaErrorNotSupported;
    GemmTcParams q = *p;
    q.m_halves = q.m_halves == 2 && (q.NTL * 16) % (2 * TS_BM) == 0 ? 2 : 1;
    const int t_max = q.m_halves == 2 ? 192 : 256;
    if (q.t_tile > t_max) q.t_tile = t_max;
    CUtensorMap map;
    cuuint64_t dims[2] = {(cuuint64_t)q.K, (cuuint64_t)q.T};
    cuuint64_t strides[1] = {(cuuint64_t)ldx * 2};
    cuuint32_t box[2] = {TS_BK, (cuuint32_t)q.t_tile};
    cuuint32_t estr[2] = {1, 1};
    if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)x, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    // K splits: of TC_EPI_STORE_F32 with planes as b2_gemm_tc_splits counts them, of the residual form in whole pairs of
    // k-blocks (a pair shares its scales)
    const bool planes = q.epi == TC_EPI_STORE_F32 && q.plane_stride > 0 && q.softcap <= 0.f;
    int ks = (q.epi == TC_EPI_RESID_F32 || planes) && q.k_splits > 1 ? (q.k_splits < q.KB ? q.k_splits : q.KB) : 1;
    int per = (q.KB + ks - 1) / ks;
    if (ks > 1 && !planes) per = (per + 1) & ~1;
    ks = (q.KB + per - 1) / per;
    const bool uni = q.gshift == 2 && (q.off32 & 3) == 0 && (ks == 1 || (per & 1) == 0);
    const int n_mt = (q.NTL * 16) / (TS_BM * q.m_halves), n_tt = (q.T + q.t_tile - 1) / q.t_tile;
    const int acc = ((q.t_tile + 31) & ~31) * q.m_halves, KS = acc <= 256 ? 2 : 1;
    // as many stages as 192 KB hold: their depth covers the latency of the loads.  (A CTA has the SM's tensor memory to
    // itself; its registers keep a second one off.)
    const int stage = q.t_tile * 128 * KS;
    int stages = TS_STAGE_SMEM / stage;
    q.stages = stages > TS_MAX_STAGES ? TS_MAX_STAGES : stages;
    const size_t smem = 1024 + (size_t)q.stages * stage + TS_PRODUCERS * TC_EPI_STAGE + (2 * q.stages + 2 * TS_SLOTS + 1) * 8 + 16;
    auto go = [&](auto kern, SmemOptIn& optin) -> int {
        if (cudaError_t e = optin.ensure(kern, smem)) return e;
        return launch_pdl(kern, dim3(n_mt * n_tt * ks), dim3((TS_PRODUCERS + 1 + q.m_halves) * 32), smem, stream, q, map, n_mt, n_tt, per);
    };
    static SmemOptIn o[6];
    if (q.m_halves == 1) return uni ? go(gemm_int4_ts_kernel<1, 2, true>, o[0]) : go(gemm_int4_ts_kernel<1, 2, false>, o[1]);
    if (KS == 2) return uni ? go(gemm_int4_ts_kernel<2, 2, true>, o[2]) : go(gemm_int4_ts_kernel<2, 2, false>, o[3]);
    return uni ? go(gemm_int4_ts_kernel<2, 1, true>, o[4]) : go(gemm_int4_ts_kernel<2, 1, false>, o[5]);
}
