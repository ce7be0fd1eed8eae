// Many-row projection in fp32: out[t][n] = sum_k x[t][k] w[n][k].  It serves models that run entirely in 32 bits.  Operands
// whose rows start on 16-byte boundaries, as an engine's do, go to the tensor cores in three bf16 terms each (csrc/gemm_f32_tc.cu);
// this file has the plan of the splits over K for both, and the kernel of fp32 FMAs for all other operands and for a short K:
//
// Bound: the FMA pipes (74 TFLOP/s).  A CTA of 128 threads owns [8 RT tokens x 128 outputs], a thread RT x 8 of them.
// Both operands are contiguous in k, so they go from global memory into shared memory as they are (cp.async, four
// stages of 16 k; rows of 20 floats, so that the 16-byte reads of 8 adjacent rows meet no bank twice) and two
// adjacent k form one packed FMA (fma.rn.f32x2): half the issue slots, and no operand has to be duplicated.  An
// output is the sum of its even-k and its odd-k chain.
// Operands reach the registers at 32 floats a clock and an 8 x 8 thread tile asks for a quarter of a float per FMA, so
// shared memory and the FMA pipes are about equally busy.  Measured in a prompt of 200 rows (12 layers of width 2048):
// 30 TFLOP/s, the whole prompt 14.5 ms; on the tensor cores 4.8 ms.
#include "gemm_f32.cuh"

#define GF_BN 128
#define GF_K 16
#define GF_LD (GF_K + 4)
#define GF_STAGES 4
#define GF_THREADS 128

// four bytes, or (valid 0) a zero
__device__ __forceinline__ void cp_async_zfill(float* dst, const float* src, int valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid) : "memory");
}
__device__ __forceinline__ void fma_x2(unsigned long long& c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

template <int RT>
__global__ void __launch_bounds__(GF_THREADS) gemm_f32_kernel(const GemmF32Params p) {
    constexpr int BT = 8 * RT;
    extern __shared__ float4 gf_smem[];
    float* ws = (float*)gf_smem;                          // [GF_STAGES][GF_BN][GF_LD]
    float* xs = ws + GF_STAGES * GF_BN * GF_LD;           // [GF_STAGES][BT][GF_LD]
    const int tid = threadIdx.x, lx = tid & 7, ly = (tid & 31) >> 3, warp = tid >> 5;
    const int t0 = blockIdx.y * BT, n0 = blockIdx.x * GF_BN;
    const int blocks = (p.K + GF_K - 1) / GF_K, per = (blocks + (int)gridDim.z - 1) / (int)gridDim.z;
    const int kb0 = (int)blockIdx.z * per, KB = max(0, min(blocks, kb0 + per) - kb0);
    // rows beyond the matrix and columns beyond K are zeros
    auto stage_rows = [&](float* dst, const float* src, int ld, int rows, int row0, int row_end, int kb) {
        for (int i = tid; i < rows * GF_K; i += GF_THREADS) {
            const int r = i / GF_K, c = i % GF_K, k = (kb0 + kb) * GF_K + c;
            const int valid = row0 + r < row_end && k < p.K ? 4 : 0;
            cp_async_zfill(dst + r * GF_LD + c, valid ? src + (size_t)(row0 + r) * ld + k : src, valid);
        }
    };
    auto stage_w = [&](int kb) { stage_rows(ws + (kb % GF_STAGES) * GF_BN * GF_LD, p.w, p.ldw, GF_BN, n0, p.N, kb); };
    auto stage_x = [&](int kb) { stage_rows(xs + (kb % GF_STAGES) * BT * GF_LD, p.x, p.ldx, BT, t0, p.T, kb); };

    pdl_launch_dependents();
    if (!p.w_older) pdl_wait();
    for (int s = 0; s < GF_STAGES - 1; ++s)
        if (s < KB) stage_w(s);
    pdl_wait();
    for (int s = 0; s < GF_STAGES - 1; ++s) {
        if (s < KB) stage_x(s);
        cp_async_commit();
    }
    // outputs of a thread: column lx of two halves of four 16-wide groups, so that it holds gate and up of the rows
    // interleaved by 8; tokens ty + 8 i
    const int wrow = (warp & 1) * 64 + lx, ty = ly + 4 * (warp >> 1);
    unsigned long long acc[RT][8];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
    for (int kb = 0; kb < KB; ++kb) {
        cp_async_wait<GF_STAGES - 2>();
        __syncthreads();                                  // block kb is here, and nobody still reads the stage of kb - 1
        if (kb + GF_STAGES - 1 < KB) { stage_w(kb + GF_STAGES - 1); stage_x(kb + GF_STAGES - 1); }
        cp_async_commit();
        const float* wb = ws + (kb % GF_STAGES) * GF_BN * GF_LD + wrow * GF_LD;
        const float* xb = xs + (kb % GF_STAGES) * BT * GF_LD + ty * GF_LD;
#pragma unroll
        for (int c = 0; c < GF_K; c += 4) {
            ulonglong2 a[RT];
#pragma unroll
            for (int i = 0; i < RT; ++i) a[i] = *(const ulonglong2*)(xb + 8 * i * GF_LD + c);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 b = *(const ulonglong2*)(wb + 8 * j * GF_LD + c);
#pragma unroll
                for (int i = 0; i < RT; ++i) { fma_x2(acc[i][j], a[i].x, b.x); fma_x2(acc[i][j], a[i].y, b.y); }
            }
        }
    }
    cp_async_wait<0>();
    const size_t plane = (size_t)blockIdx.z * (size_t)p.plane_stride;
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int t = t0 + ty + 8 * i;
        if (t >= p.T) continue;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __uint_as_float((unsigned)acc[i][j]) + __uint_as_float((unsigned)(acc[i][j] >> 32));
        if (p.mode == DG_GATE_PAIR) {
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const int n = n0 + wrow + 8 * j, o = (n >> 4) * 8 + (n & 7);
                if (n + 8 < p.N) ((float*)p.out)[(size_t)t * p.ldo + o] = (p.act == ACT_RELU ? fmaxf(v[j], 0.f) : silu_p(v[j])) * v[j + 1];
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int n = n0 + wrow + 8 * j;
                if (n < p.N)
                    ((float*)p.out)[(size_t)t * p.ldo + n + plane] =
                        (p.mode == DG_STORE_F32 && p.softcap > 0.f) ? p.softcap * tanhf(v[j] / p.softcap)
                                                                    : (p.mode == DG_STORE && n < p.act_cols ? silu_p(v[j]) : v[j]);
            }
        }
    }
}

template <int RT>
static int launch_f32(const GemmF32Params* p, int splits, cudaStream_t s) {
    constexpr size_t smem = (size_t)GF_STAGES * (GF_BN + 8 * RT) * GF_LD * 4;
    static SmemOptIn optin;
    if (cudaError_t e = optin.ensure(gemm_f32_kernel<RT>, smem)) return e;
    const dim3 grid((p->N + GF_BN - 1) / GF_BN, (p->T + 8 * RT - 1) / (8 * RT), splits);
    return launch_pdl(gemm_f32_kernel<RT>, grid, dim3(GF_THREADS), smem, s, *p);
}

// Splits over K with the least time on the busiest SM: a 64-k block of t <= 128 tokens takes a tensor-core CTA about 0.95 +
// 0.003 t us (9 tokens 1.0, 128 tokens 1.3), a start and an end 5, a further plane 1 in its consumer; whole waves of CTAs.
static int tc_tile_f32(int T) { const int n = (T + 127) / 128; return ((T + n - 1) / n + 15) & ~15; }
B2_API int b2_gemm_f32_splits(int N, int K, int T, int max_splits) {
    const int t = tc_tile_f32(T), ctas = (N + 127) / 128 * ((T + t - 1) / t), blocks = (K + 63) / 64;
    int best = 1;
    double least = 1e30;
    for (int want = 1; want <= (max_splits < 1 ? 1 : max_splits); ++want) {
        const int per = (blocks + want - 1) / want, ks = (blocks + per - 1) / per, waves = (ctas * ks + 147) / 148;      // no split is empty
        const double cost = waves * (per * (0.95 + 0.003 * t) + 5.0) + (ks - 1);
        if (cost < least - 1e-9) { least = cost; best = ks; }
    }
    return best;
}

// p->max_splits > 1 (DG_STORE_F32 without a cap): the product may be split over K; split z stores its own plane,
// plane_stride floats apart (b2_gemm_f32_splits tells how many there are).
B2_API int b2_gemm_f32(const GemmF32Params* p, cudaStream_t s) {
    if (p->T < 1 || p->N < 1 || p->K < 1 || p->ldx < p->K || p->ldw < p->K) return cudaErrorInvalidValue;
    if (p->mode == DG_GATE_PAIR && (p->N & 15)) return cudaErrorInvalidValue;
    const bool planes = p->mode == DG_STORE_F32 && p->softcap <= 0.f && p->plane_stride > 0;
    const int ks = b2_gemm_f32_splits(p->N, p->K, p->T, planes && p->max_splits > 1 ? p->max_splits : 1);
    // A short K is over before the tensor-core CTA is set up: with one FMA CTA an SM at most, K = 32 3.9 to 5.5 us against 4.8 to 7.7 (9 to 500
    // rows), K = 64 and 128 rows of 512 outputs 6.2 against 7.5; but K = 64, 33 rows 6.2 and 6.1, 128 rows of 2048 outputs 8.4 and 7.7
    const long long fma_ctas = (long long)((p->N + GF_BN - 1) / GF_BN) * ((p->T + 15) / 16);
    const bool brief = (p->K <= 32 && fma_ctas <= 148) || (p->K <= 64 && p->T > 64 && fma_ctas <= 64);
    if (!brief && !((p->ldx | p->ldw) & 3) && !(((uintptr_t)p->x | (uintptr_t)p->w) & 15)) return gemm_f32_tc_launch(p, tc_tile_f32(p->T), ks, s);
    // Tokens of an FMA CTA (8 rt): us a 16-k block with n CTAs on an SM, about 0.5 + s n, s = .38, .54, .62, .73, .85, 1.02 for
    // rt = 2, 4, 5, 6, 7, 8 (one CTA alone does not cover its own latencies)
    static const double slope[9] = {0, 0, 0.38, 0, 0.54, 0.62, 0.73, 0.85, 1.02};
    int rt = 8;
    double least = 1e30;
    for (int r = 8; r >= 2; --r) {
        if (r == 3) continue;
        const int n = ((p->N + GF_BN - 1) / GF_BN * ((p->T + 8 * r - 1) / (8 * r)) * ks + 147) / 148;
        const double cost = 0.5 + slope[r] * n;
        if (cost < least - 1e-9) { least = cost; rt = r; }
    }
    switch (rt) {
        case 2: return launch_f32<2>(p, ks, s);
        case 4: return launch_f32<4>(p, ks, s);
        case 5: return launch_f32<5>(p, ks, s);
        case 6: return launch_f32<6>(p, ks, s);
        case 7: return launch_f32<7>(p, ks, s);
        default: return launch_f32<8>(p, ks, s);
    }
}
B2_API int b2_sizeof_gemm_f32_params() { return (int)sizeof(GemmF32Params); }
