// Many-row projection in fp32 on the tensor cores, without giving up a bit of an operand: out[t][n] = sum_k x[t][k] w[n][k].
//
// An fp32 number is the sum of three bf16 numbers (8 + 8 + 8 bits): w = w0 + w1 + w2, x = x0 + x1 + x2.  Of the nine products
// the six that are not below the last bit are formed by tcgen05.mma kind::f16, which multiplies bf16 exactly:
// w0 x0 + (w0 x1 + w1 x0) + (w0 x2 + w1 x1 + w2 x0), the smallest first.  Where the 128 x 64 weights of a block are bf16 numbers
// (a bf16 checkpoint run in 32 bits), w1 and w2 are zero, and their three products are left out.
// bf16 has the exponents of fp32, so the third term of a number below 2^-110 would lie among its subnormals or below them: both
// operands are split times 2^24, which loses nothing and costs 1 % of the time (weights that need all 24 bits 3 %).  Numbers above
// 2^103 and sums above 2^79 become infinite by that and are formed again, see below.
// The tensor core cuts its sums off where fp32 additions round, so it never sums more than one block of 64 k: every block starts
// from zero in tensor memory, and the warps add the blocks' sums in registers.  Error against 64 bits (2-norms, 200 rows,
// K = 2048 / 6144): 1.3e-7 / 1.95e-7; two chains of fp32 FMAs, as before: 5.7e-7 / 9.9e-7.
//
// A CTA owns [128 outputs x t_tile <= 128 tokens].  TMA brings the fp32 operands of a block (two stages).  All 16 worker
// warps do the same per block: split 16 weights a lane, which go from registers into tensor memory as the A operand
// (tcgen05.st 16x128b; a lane takes 16 bytes of a row, so the k of a 16-group are permuted, in both operands alike), split 16
// activations a lane into shared memory (B operand, 128-byte swizzle), then take in the block before.  Two stages here too: one
// is multiplied while the other is split.
// Bound: the splitting and what surrounds it, 490 instructions a warp and block with weights of 24 bits (63 % of the issue slots
// at 200 rows, 2048 -> 8736; tensor pipe 42 % of the time).  That shape takes 46 us (53 with weights that need all 24 bits), FMAs 245;
// 128 rows, 8192 -> 18944: 172 (232), FMAs 1132 us.
// A result that is not finite is formed again by fp32 FMAs (ft_again): infinities and numbers that no bf16 reaches come out as they do there.
// Every mbarrier wait is bounded; on expiry a CTA records a status and forms its outputs by fp32 FMAs.
#include <cuda.h>
#include <cuda_bf16.h>
#include "mixers.cuh"
#include "tc_util.cuh"
#include "gemm_f32.cuh"

#define FT_WARPS 16
#define FT_THREADS ((FT_WARPS + 2) * 32)
#define FT_BK 64
#define FT_BM 128
#define FT_BT 128
#define FT_PLANE (FT_BT * 128)               // bytes of a term of the activations in a stage
#define FT_STAGE (3 * FT_PLANE)
#define FT_RAW (2 * (FT_BM + FT_BT) * 128)    // fp32 operands of a block: two boxes of 32 k each
#define FT_SMEM (1024 + 2 * FT_STAGE + 2 * FT_RAW)
#define FT_SCALE 16777216.f                  // both operands are split times 2^24, the sums of a block taken in times 2^-48 (exact)

__device__ __forceinline__ void ft_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        :: "r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void ft_store(uint32_t a, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "r"(a), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ uint32_t ft_scale2(uint32_t two) {
    const __nv_bfloat162 b = __hmul2(*(const __nv_bfloat162*)&two, __float2bfloat162_rn(FT_SCALE));
    return *(const uint32_t*)&b;
}
// the next bf16 term of two numbers, which are left with what it does not hold
__device__ __forceinline__ uint32_t ft_term(float& x, float& y) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
    const uint32_t u = *(const uint32_t*)&b;
    x -= __uint_as_float(u << 16);
    y -= __uint_as_float(u & 0xffff0000u);
    return u;
}
// (of all worker warps; also a barrier among them)
__device__ __forceinline__ bool ft_any_worker(bool mine) {
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, %2, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
                 : "=r"(any) : "r"((uint32_t)mine), "n"(FT_WARPS * 32) : "memory");
    return any != 0;
}
__device__ __forceinline__ void ft_copy16(unsigned char* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
// The results marked in `again` (bit c: acc[c], token t0 + c0 + c of output n) once more, as chains of fp32 FMAs over
// k_lo .. k_hi - 1.  All worker warps take part: both operands pass through the shared memory that held their raw blocks, two blocks of
// 64 k in turn, a row's 16-byte pieces permuted by its number (lanes read one piece of 32 rows without conflicts).  Bound: a few
// results the staging, many the reads of x, which all lanes make alike.  128 rows, 6144 -> 2048: one row of NaN 306 us, all rows
// 2.2 ms (a lane's chain straight from global memory: 1.0 and 93 ms; the product by FMAs, which needs no second pass, 309 us).
__device__ __forceinline__ void ft_again(const GemmF32Params& p, unsigned char* buf, float* keep, volatile int* abort_flag, float (&acc)[32], uint32_t again, int n, int row,
                                         int n0, int t0, int t_tile, int c0, int k_lo, int k_hi, int tid) {
    if (*abort_flag) {                       // copies may still be on their way to shared memory
#pragma unroll
        for (int c = 0; c < 32; ++c) {
            if (!(again >> c & 1)) continue;
            const float *xt = p.x + (size_t)(t0 + c0 + c) * p.ldx, *wn = p.w + (size_t)n * p.ldw;
            float v = 0.f;
#pragma unroll 1
            for (int k = k_lo; k < k_hi; ++k) v = fmaf(xt[k], wn[k], v);
            acc[c] = v;
        }
        return;
    }
    const uint32_t of_warp = __reduce_or_sync(0xffffffffu, again);
    auto stage = [&](int b) {
        for (int i = tid; i < (FT_BM + t_tile) * 16; i += FT_WARPS * 32) {
            const int r = i >> 4, ch = i & 15, k = k_lo + b * FT_BK + 4 * ch, g = r < FT_BM ? n0 + r : t0 + r - FT_BM;
            const int bytes = g < (r < FT_BM ? p.N : p.T) ? 4 * max(0, min(4, k_hi - k)) : 0;
            const float* src = r < FT_BM ? p.w + (size_t)g * p.ldw + k : p.x + (size_t)g * p.ldx + k;
            ft_copy16(buf + (b & 1) * FT_RAW + r * 256 + ((ch ^ (r & 7)) << 4), bytes ? src : p.w, bytes);
        }
        cp_async_commit();
    };
    auto fma4 = [](const float4& x, const float4& w, float v) { return fmaf(x.w, w.w, fmaf(x.z, w.z, fmaf(x.y, w.y, fmaf(x.x, w.x, v)))); };
    const int blocks = (k_hi - k_lo + FT_BK - 1) / FT_BK;
    constexpr int LD = FT_WARPS * 32;        // results and sums wait in shared memory, a column a thread
#pragma unroll
    for (int c = 0; c < 32; ++c) keep[c * LD] = (again >> c & 1) ? 0.f : acc[c];
    stage(0);
#pragma unroll 1
    for (int b = 0; b < blocks; ++b) {
        if (b + 1 < blocks) stage(b + 1); else cp_async_commit();
        cp_async_wait<1>();
        ft_any_worker(false);
        const unsigned char* wr = buf + (b & 1) * FT_RAW + row * 256;
        const unsigned char* xr = buf + (b & 1) * FT_RAW + (FT_BM + c0) * 256;      // (c0 is a multiple of 32)
#pragma unroll 1
        for (int h = 0; h < 32; h += 8) {
            uint32_t m = of_warp >> h & 0xffu;
            if (__popc(m) > 2) {             // most of the eight: all of them
                float v[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) v[c] = keep[(h + c) * LD];
#pragma unroll 2
                for (int ch = 0; ch < FT_BK / 4; ++ch) {
                    const float4 w = *(const float4*)(wr + ((ch ^ (row & 7)) << 4));
#pragma unroll
                    for (int c = 0; c < 8; ++c) v[c] = fma4(*(const float4*)(xr + (h + c) * 256 + ((ch ^ c) << 4)), w, v[c]);
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) if (again >> (h + c) & 1) keep[(h + c) * LD] = v[c];
            } else
                for (; m; m &= m - 1) {
                    const int c = __ffs(m) - 1;
                    float v = keep[(h + c) * LD];
#pragma unroll 4
                    for (int ch = 0; ch < FT_BK / 4; ++ch)
                        v = fma4(*(const float4*)(xr + (h + c) * 256 + ((ch ^ c) << 4)), *(const float4*)(wr + ((ch ^ (row & 7)) << 4)), v);
                    if (again >> (h + c) & 1) keep[(h + c) * LD] = v;
                }
        }
        ft_any_worker(false);                // (the block is read before it is overwritten)
    }
    cp_async_wait<0>();
#pragma unroll
    for (int c = 0; c < 32; ++c) acc[c] = keep[c * LD];
}
__global__ void __launch_bounds__(FT_THREADS, 1) gemm_f32_tc_kernel(const GemmF32Params p, const __grid_constant__ CUtensorMap wmap,
                                                                     const __grid_constant__ CUtensorMap xmap, const int t_tile, const int per_kb) {
    extern __shared__ __align__(1024) unsigned char ft_smem[];
    unsigned char* sB = (unsigned char*)(((uintptr_t)ft_smem + 1023) & ~(uintptr_t)1023);       // [2][3][128 tokens of 128 bytes]
    unsigned char* sR = sB + 2 * FT_STAGE;                                                      // [2][weights: 2 boxes | activations: 2 boxes]
    __shared__ uint64_t raw_full[2];         // the fp32 operands have arrived (TMA bytes)
    __shared__ uint64_t raw_empty[2];        // they have been read: one arrival per worker warp
    __shared__ uint64_t full[2];             // operands of the stage are in place: one arrival per worker warp
    __shared__ uint64_t done[2];             // the block is multiplied: its stage is free and its sums can be read (commit)
    __shared__ uint32_t s_tmem, s_terms[2];  // s_terms: number + 1 of the last block of the stage whose weights have a second or third term
    __shared__ int s_abort;
    volatile int* abort_flag = &s_abort;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int n0 = blockIdx.x * FT_BM, t0 = blockIdx.y * t_tile;
    const int blocks = (p.K + FT_BK - 1) / FT_BK, kb0 = (int)blockIdx.z * per_kb, KB = min(blocks - kb0, per_kb);
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], FT_WARPS);
            mbar_init(&full[s], FT_WARPS); mbar_init(&done[s], 1); s_terms[s] = 0;
        }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == FT_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // tensor memory: sums of the two stages (128 columns each), then their weights, 32 columns a term
    const uint32_t tmem = s_tmem, tmem_a = tmem + 256;
    pdl_launch_dependents();                 // (every CTA has its tensor memory)
    if (warp < FT_WARPS) {
        // weights: rows g and g + 8 of tile rt, k half kh of a block; activations: 16 k from 16 m of token tok
        const int rt = 2 * (warp & 3) + ((warp >> 2) & 1), kh = warp >> 3, g = lane >> 2, t = lane & 3;
        const int tok = warp * 8 + (lane & 7), m = lane >> 3;
        const bool has_x = tok < t_tile;
        const unsigned char* raw_a = sR + kh * (FT_BM * 128) + (rt * 16 + g) * 128;
        const unsigned char* raw_x = sR + 2 * (FT_BM * 128) + (m >> 1) * (FT_BT * 128) + tok * 128;
        float acc[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) acc[c] = 0.f;
        const int c0 = (warp >> 2) * 32;     // this warp's tokens of the tile; its outputs are lanes 32 (warp & 3) ..
        const uint32_t t_ld = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
        const uint32_t t_st = tmem_a + ((uint32_t)(rt * 16) << 16) + (uint32_t)(kh * 16);
        unsigned char* b_row = sB + tok * 128;
        bool ok = true;
        // wait for a barrier: one lane polls
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
            int o = 1;
            if (lane == 0) o = mbar_wait(bar, parity, abort_flag) ? 1 : 0;
            return __shfl_sync(0xffffffffu, o, 0) != 0;
        };
        // the second and third terms of the weights lie in tensor memory only where there are any: zeros[s] says that this
        // warp's part of stage s holds zeros
        bool zeros[2] = {false, false};
        for (int kb = 0; kb <= KB; ++kb) {
            const int s = kb & 1;
            if (kb < KB) {
                // (stage s is free: this warp has taken in block kb - 2)
                ok = wait(&raw_full[s], (kb >> 1) & 1);
                if (!ok) break;
                float4 a[4], x[4];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const unsigned char* r = raw_a + s * FT_RAW + (((4 * j + t) ^ g) << 4);
                    a[2 * j] = *(const float4*)r;
                    a[2 * j + 1] = *(const float4*)(r + 8 * 128);
                }
                if (has_x) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) x[q] = *(const float4*)(raw_x + s * FT_RAW + (((4 * (m & 1) + q) ^ (tok & 7)) << 4));
                }
                uint32_t low = 0;                  // any bit that the first term does not hold
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    low |= __float_as_uint(a[j].x) | __float_as_uint(a[j].y) | __float_as_uint(a[j].z) | __float_as_uint(a[j].w);
                const bool rest = __any_sync(0xffffffffu, (low & 0xffffu) != 0);
                uint32_t r[8];
                if (!rest) {                       // bf16 numbers: their upper halves
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int e = 4 * (j >> 1) + (j & 1);
                        r[e] = ft_scale2(__byte_perm(__float_as_uint(a[j].x), __float_as_uint(a[j].y), 0x7632));
                        r[e + 2] = ft_scale2(__byte_perm(__float_as_uint(a[j].z), __float_as_uint(a[j].w), 0x7632));
                    }
                    ft_store(t_st + (uint32_t)(s * 96), r);
                    if (!(s ? zeros[1] : zeros[0])) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) r[e] = 0u;
                        ft_store(t_st + (uint32_t)(s * 96 + 32), r);
                        ft_store(t_st + (uint32_t)(s * 96 + 64), r);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) { a[j].x *= FT_SCALE; a[j].y *= FT_SCALE; a[j].z *= FT_SCALE; a[j].w *= FT_SCALE; }
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int e = 4 * (j >> 1) + (j & 1);
                            r[e] = ft_term(a[j].x, a[j].y);
                            r[e + 2] = ft_term(a[j].z, a[j].w);
                        }
                        ft_store(t_st + (uint32_t)(s * 96 + i * 32), r);
                    }
                }
                if (s) zeros[1] = !rest; else zeros[0] = !rest;
                if (rest && lane == 0) s_terms[s] = (uint32_t)(kb + 1);
                if (has_x) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) { x[q].x *= FT_SCALE; x[q].y *= FT_SCALE; x[q].z *= FT_SCALE; x[q].w *= FT_SCALE; }
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        uint4 lo, hi;
                        lo.x = ft_term(x[0].x, x[0].y); lo.y = ft_term(x[1].x, x[1].y); lo.z = ft_term(x[2].x, x[2].y); lo.w = ft_term(x[3].x, x[3].y);
                        hi.x = ft_term(x[0].z, x[0].w); hi.y = ft_term(x[1].z, x[1].w); hi.z = ft_term(x[2].z, x[2].w); hi.w = ft_term(x[3].z, x[3].w);
                        unsigned char* b = b_row + s * FT_STAGE + i * FT_PLANE;
                        const int c = 2 * m;
                        *(uint4*)(b + (((c) ^ (tok & 7)) << 4)) = lo;
                        *(uint4*)(b + (((c + 1) ^ (tok & 7)) << 4)) = hi;
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                fence_proxy_async_smem();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { mbar_arrive(&full[s]); mbar_arrive(&raw_empty[s]); }
            }
            if (kb > 0) {
                ok = wait(&done[s ^ 1], ((kb - 1) >> 1) & 1);
                if (!ok) break;
                tc_fence_after();
                if (c0 < t_tile) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t r[16];
                        tc_ld16(t_ld + (uint32_t)((s ^ 1) * 128 + h * 16), r);
                        tc_wait_ld();
#pragma unroll
                        for (int c = 0; c < 16; ++c) acc[h * 16 + c] = fmaf(__uint_as_float(r[c]), 1.f / (FT_SCALE * FT_SCALE), acc[h * 16 + c]);
                    }
                }
                tc_fence_before();
            }
        }
        // ---- epilogue: a lane has one output of 32 tokens
        const int n = n0 + (warp & 3) * 32 + lane, nt = min(32, min(t_tile, p.T - t0) - c0);      // (tokens of this warp; none if negative)
        pdl_wait();
        uint32_t again = 0;                  // tokens whose result is not finite (or, if a wait expired, all)
        if (n < p.N) {
#pragma unroll
            for (int c = 0; c < 32; ++c) if (c < nt && (!ok || !isfinite(acc[c]))) again |= 1u << c;
        }
        if (ft_any_worker(again != 0)) ft_again(p, sR, (float*)sB + tid, abort_flag, acc, again, n, (warp & 3) * 32 + lane, n0, t0, t_tile, c0, kb0 * FT_BK, min(p.K, (kb0 + KB) * FT_BK), tid);
        const size_t plane = (size_t)blockIdx.z * (size_t)p.plane_stride;
        if (p.mode == DG_GATE_PAIR) {
            float* out = (float*)p.out + (size_t)(t0 + c0) * p.ldo + (n >> 4) * 8 + (n & 7);
            const bool mine = !(lane & 8) && n + 8 < p.N;
#pragma unroll
            for (int c = 0; c < 32; ++c) {
                const float up = __shfl_down_sync(0xffffffffu, acc[c], 8);
                if (mine && c < nt) out[(size_t)c * p.ldo] = (p.act == ACT_RELU ? fmaxf(acc[c], 0.f) : silu_p(acc[c])) * up;
            }
        } else if (n < p.N) {
            if (p.mode == DG_STORE_F32 && p.softcap > 0.f) {
#pragma unroll
                for (int c = 0; c < 32; ++c) acc[c] = p.softcap * tanhf(acc[c] / p.softcap);
            } else if (p.mode == DG_STORE && n < p.act_cols) {
#pragma unroll
                for (int c = 0; c < 32; ++c) acc[c] = silu_p(acc[c]);
            }
            float* out = (float*)p.out + (size_t)(t0 + c0) * p.ldo + n + plane;
#pragma unroll
            for (int c = 0; c < 32; ++c) if (c < nt) out[(size_t)c * p.ldo] = acc[c];
        }
    } else if (warp == FT_WARPS + 1) {
        // ---- fp32 operands; the weights of the first two blocks need not wait for the kernel before this one
        const uint32_t bytes = 2 * FT_BM * 128 + 2 * (uint32_t)t_tile * 128;
        if (!p.w_older) pdl_wait();
        for (int kb = -2; kb < KB; ++kb) {
            // block b: all of it, or (the first two, in two steps) its weights or its activations
            const int b = kb < 0 ? kb + 2 : kb, s = b & 1, k = (kb0 + b) * FT_BK;
            if (b >= KB) continue;
            if (kb == 0) pdl_wait();
            if (kb >= 2 && !__all_sync(0xffffffffu, mbar_wait(&raw_empty[s], ((kb >> 1) & 1) ^ 1, abort_flag))) break;
            if (elect_one()) {
                unsigned char* r = sR + s * FT_RAW;
                if (kb < 0 || kb >= 2) {
                    mbar_arrive_expect_tx(&raw_full[s], bytes);
                    tma_load_2d(r, &wmap, k, n0, &raw_full[s]);
                    tma_load_2d(r + FT_BM * 128, &wmap, k + 32, n0, &raw_full[s]);
                }
                if (kb >= 0) {
                    tma_load_2d(r + 2 * FT_BM * 128, &xmap, k, t0, &raw_full[s]);
                    tma_load_2d(r + 2 * FT_BM * 128 + FT_BT * 128, &xmap, k + 32, t0, &raw_full[s]);
                }
            }
            __syncwarp();
        }
    } else {
        const uint32_t idesc = make_idesc_f16(t_tile) | TC_IDESC_BF16;
        const uint64_t bd0 = make_desc_sw128(smem_u32(sB));
        for (int kb = 0; kb < KB; ++kb) {
            const int s = kb & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (kb >> 1) & 1, abort_flag))) break;
            tc_fence_after();
            const bool terms = *(volatile uint32_t*)&s_terms[s] == (uint32_t)(kb + 1);
            const uint32_t d = tmem + s * 128, a = tmem_a + s * 96;
            const uint64_t b = bd0 + (uint64_t)(s * (FT_STAGE >> 4));
            __syncwarp();
            if (elect_one()) {
                // terms (weight, activation), the smallest products first
                auto products = [&](int i, int j, uint32_t first) {
#pragma unroll
                    for (int k16 = 0; k16 < FT_BK / 16; ++k16)
                        ft_mma(d, a + 32 * i + 8 * k16, b + (uint64_t)(j * (FT_PLANE >> 4) + 2 * k16), idesc, first && k16 == 0 ? 0u : 1u);
                };
                products(0, 2, 1u);
                if (terms) { products(2, 0, 0u); products(1, 1, 0u); products(1, 0, 0u); }
                products(0, 1, 0u);
                products(0, 0, 0u);
                tc_commit(&done[s]);
            }
            __syncwarp();
        }
    }
    if (s_abort && tid == 0 && p.status) atomicExch(p.status, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == FT_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512) : "memory");
}

int gemm_f32_tc_launch(const GemmF32Params* p, int t_tile, int splits, cudaStream_t s) {
    static SmemOptIn optin;
    if (cudaError_t e = optin.ensure(gemm_f32_tc_kernel, FT_SMEM)) return e;
    EncodeTiledFn enc = get_encode();
    if (!enc) return cudaErrorNotSupported;
    auto encode = [&](CUtensorMap* m, const float* base, int rows, int ld, int box_rows) {
        const cuuint64_t dims[2] = {(cuuint64_t)p->K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 4};
        const cuuint32_t box[2] = {32, (cuuint32_t)box_rows}, estr[2] = {1, 1};
        return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    CUtensorMap wmap, xmap;
    if (!encode(&wmap, p->w, p->N, p->ldw, FT_BM) || !encode(&xmap, p->x, p->T, p->ldx, t_tile)) return cudaErrorInvalidValue;
    const int blocks = (p->K + FT_BK - 1) / FT_BK, per = (blocks + splits - 1) / splits;
    const dim3 grid((p->N + FT_BM - 1) / FT_BM, (p->T + t_tile - 1) / t_tile, (blocks + per - 1) / per);
    return launch_pdl(gemm_f32_tc_kernel, grid, dim3(FT_THREADS), FT_SMEM, s, *p, wmap, xmap, t_tile, per);
}
