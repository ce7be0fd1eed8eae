// Epilogue of the tcgen05 GEMMs (csrc/gemm_int4.cu, csrc/gemm_tc.cu): what becomes of 16 token columns of 32 outputs that a
// warp has read from its tensor-memory lanes.
//
// A lane has one output of 16 tokens, and a token's outputs lie side by side in memory: the values go through 2 KB of shared
// memory of the warp's own and leave as 16 bytes a lane.  Stores of two bytes a lane took about 11 cycles each, whatever the
// tile, which was a fifth of the time of a [128 x 256] tile over 5120 k.
#pragma once
#include <cuda_bf16.h>
#include "gemm_tc.cuh"

#define TC_EPI_COLS 16
#define TC_EPI_STAGE 2048        // bytes of shared memory a warp

// 16 rows (tokens tt0 ..) of 8 << BITS 16-bit outputs from o0 on, from the warp's shared memory to where they belong
template <int BITS>
__device__ __forceinline__ void tc_rows16(const GemmTcParams& p, int lane, int o0, int tt0, int tn, const void* stage) {
    const bool vec = ((p.ldo & 7) | ((uintptr_t)p.out & 15)) == 0;
    const int o = o0 + (lane & ((1 << BITS) - 1)) * 8;
    uint16_t* dst = (uint16_t*)p.out + (size_t)(tt0 + (lane >> BITS)) * p.ldo + o;
    if (vec && o + 8 <= p.n_valid) {
#pragma unroll
        for (int j = 0; j < 1 << (BITS - 1); ++j) {
            const uint4 v = ((const uint4*)stage)[32 * j + lane];
            if ((32 >> BITS) * j + (lane >> BITS) < tn) *(uint4*)(dst + (size_t)((32 >> BITS) * j) * p.ldo) = v;
        }
    } else {
#pragma unroll 1
        for (int j = 0; j < 1 << (BITS - 1); ++j)
#pragma unroll 1
            for (int e = 0; e < 8; ++e)
                if ((32 >> BITS) * j + (lane >> BITS) < tn && o + e < p.n_valid)
                    dst[(size_t)((32 >> BITS) * j) * p.ldo + e] = ((const uint16_t*)stage)[(32 * j + lane) * 8 + e];
    }
}

// r[c]: output nb + lane of token tt0 + c, c < tn; plane: float offset of the K split (TC_EPI_STORE_F32); split: other CTAs
// add to the same residual rows; stage: the warp's shared memory.
__device__ __forceinline__ void tc_epilogue(const GemmTcParams& p, uint32_t (&r)[TC_EPI_COLS], int lane, int nb, int tt0, int tn, size_t plane,
                                            bool split, void* stage) {
    const int n = nb + lane;
    if (p.epi == TC_EPI_PUSH_F32) {
        // plain stores into the owner's memory over NVLink (posted writes, 128 bytes per warp)
        const size_t poff = (size_t)((*p.epoch + 1u) & 1u) * (size_t)p.part_stride;
#pragma unroll 4
        for (int c = 0; c < TC_EPI_COLS; ++c) {
            if (c < tn && n < p.n_valid) {
                const unsigned e = (unsigned)(tt0 + c) * (unsigned)p.ldo + (unsigned)n;
                const unsigned i4 = e >> 2, owner = i4 / p.push_per;
                float* dst = p.push[owner] + poff + ((size_t)p.push_rank * p.push_per + (i4 - owner * p.push_per)) * 4 + (e & 3u);
                *dst = __uint_as_float(r[c]);
            }
        }
        return;
    }
    if (p.epi == TC_EPI_SILU_PAIR) {
        // gate and up rows alternate by 8: of the 16 tokens of a pair of rows the gate's lane takes the first 8, the up's the
        // others, so that all lanes have products to form (the SiLU of a [256 x 80] tile by half of the lanes took 2 us more)
        const bool is_up = (lane & 8) != 0;
        const int o = (lane >> 4) * 8 + (lane & 7), c0 = is_up ? 8 : 0;
        float v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float mine = __uint_as_float(is_up ? r[c + 8] : r[c]);
            const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(is_up ? r[c] : r[c + 8]), 8);
            const float gate = is_up ? other : mine, up = is_up ? mine : other;
            v[c] = (p.act ? fmaxf(gate, 0.f) : silu_f(gate)) * up;
        }
        if (p.bf16) {
#pragma unroll
            for (int c = 0; c < 8; ++c) ((__nv_bfloat16*)stage)[(c0 + c) * 16 + o] = __float2bfloat16(v[c]);
        } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) ((__half*)stage)[(c0 + c) * 16 + o] = __float2half(v[c]);
        }
        __syncwarp();
        tc_rows16<1>(p, lane, nb / 2, tt0, tn, stage);
        __syncwarp();
        return;
    }
    if (p.epi == TC_EPI_STORE_F16) {
        if (n < p.act_cols) {
#pragma unroll
            for (int c = 0; c < TC_EPI_COLS; ++c) r[c] = __float_as_uint(silu_f(__uint_as_float(r[c])));
        }
        if (p.bf16) {
#pragma unroll
            for (int c = 0; c < TC_EPI_COLS; ++c) ((__nv_bfloat16*)stage)[c * 32 + lane] = __float2bfloat16(__uint_as_float(r[c]));
        } else {
#pragma unroll
            for (int c = 0; c < TC_EPI_COLS; ++c) ((__half*)stage)[c * 32 + lane] = __float2half(__uint_as_float(r[c]));
        }
        __syncwarp();
        tc_rows16<2>(p, lane, nb, tt0, tn, stage);
        __syncwarp();
        return;
    }
    float* s = (float*)stage;
    float* out = (float*)p.out + (p.epi == TC_EPI_STORE_F32 ? plane : 0);
    const bool vec = ((p.ldo & 3) | ((uintptr_t)out & 15)) == 0, resid = p.epi != TC_EPI_STORE_F32;
    if (!resid && p.softcap > 0.f) {
#pragma unroll
        for (int c = 0; c < TC_EPI_COLS; ++c) r[c] = __float_as_uint(p.softcap * tanhf(__uint_as_float(r[c]) / p.softcap));
    }
#pragma unroll
    for (int c = 0; c < TC_EPI_COLS; ++c) s[c * 32 + lane] = __uint_as_float(r[c]);
    __syncwarp();
    const int o = nb + (lane & 7) * 4;
    float* dst = out + (size_t)(tt0 + (lane >> 3)) * p.ldo + o;
    const size_t row4 = (size_t)4 * p.ldo;
    if (vec && o + 4 <= p.n_valid) {
        if (resid && !split) {
            float4 old[4];                         // (requested together: stores between the loads would keep them apart)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (4 * j + (lane >> 3) < tn) old[j] = *(const float4*)(dst + j * row4);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 v = ((const float4*)s)[j * 32 + lane];
                if (4 * j + (lane >> 3) < tn) *(float4*)(dst + j * row4) = make_float4(v.x + old[j].x, v.y + old[j].y, v.z + old[j].z, v.w + old[j].w);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 v = ((const float4*)s)[j * 32 + lane];
                if (4 * j + (lane >> 3) >= tn) continue;
                if (resid) atomicAdd((float4*)(dst + j * row4), v);
                else *(float4*)(dst + j * row4) = v;
            }
        }
    } else {
#pragma unroll 1
        for (int j = 0; j < 4; ++j)
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                if (4 * j + (lane >> 3) >= tn || o + k >= p.n_valid) continue;
                float* d = dst + j * row4 + k;
                const float v = s[(j * 32 + lane) * 4 + k];
                if (!resid) *d = v;
                else if (split) atomicAdd(d, v);
                else *d += v;
            }
    }
    __syncwarp();
}
