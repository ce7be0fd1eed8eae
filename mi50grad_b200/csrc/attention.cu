// Decode / verify attention with a KV cache: split-KV flash decoding with an
// in-kernel merge, a sigmoid output gate and optional draft-tree masks.
//
// One kernel covers the reference's decode attention, its sigmoid gate and its
// tree-masked variant (reference: src/kernels/flash_attn_256_tuned.hip:171-350,
// src/kernels/sigmoid_mul.hip:10, src/kernels/flash_attn_tree.hip:74-193), with
// per-row sequence ids, lengths and masks read from device memory (RowMeta)
// instead of host-patched arguments.  Visibility of cache slot s for a row:
//     s < ctx   or   (s - ctx < 64 and mask bit (s - ctx) set).
//
// grid = (kv_heads, rows, splits); a CTA handles every query head of its KV head (GQA), so K/V are read
// once per group.  Each warp takes 16 cache slots at a time and multiplies them on the tensor cores with the
// heads as the narrow side: S^T = K Q^T is [16 slots x 8 heads] and O^T += V^T P^T [16 dims x 8 heads] a
// mma.sync m16n8k16, so up to eight heads cost one column tile and no shuffles but those of the running
// maximum.  The soft-max weights enter the second product as the sum of two fp16 terms; the largest is 2^15, so that
// both terms of weights down to 2^-18 of it are normal numbers (23 bits) and what falls off at the bottom is below 2^-40 of it.
// Everything else in the products is fp16 already.  The tensor core cuts off the bits below its 24 at every addition, so
// a product's own 16 terms are all that it adds up; the sums over the head dim and over the slots are fp32 additions,
// which round.  (max, sum, O) are merged across warps in shared memory and across splits through a scratch buffer by
// the last CTA to arrive.
//
// Bound: the cache, and with short contexts the latency of one pass.  With dot products on the FMA pipes a
// slot cost about 180 warp instructions for six heads (here 10), which was the bound.  Measured per layer,
// 5 sequences of 7000 slots, 4 KV heads of 256, 5 query heads each (143 MB), inside the step: 62 us against 121 (60 with sums on the tensor core).
#include "kernels.cuh"

#define ATT_WARPS 4
#define ATT_THREADS (ATT_WARPS * 32)
#define ATT_MAX_G 8
#define ATT_SLOTS 16             // cache slots a warp takes at a time
#define ATT_MIN_SPLIT_LEN (ATT_WARPS * ATT_SLOTS)      // one pass of one CTA
#define ATT_WEIGHT 32768.f       // soft-max weight of a score that is the maximum
#define ATT_LDH(HD) ((HD) + 8)   // halfs per staged row: the 16-byte rows of a matrix meet no bank twice

__device__ __forceinline__ void at_ldsm4(uint32_t (&r)[4], const __half* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void at_ldsm4_t(uint32_t (&r)[4], const __half* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void at_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t at_transpose(uint32_t x) {      // 8 x 8 matrix of 16-bit values over the warp
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}

template <int HD>
__global__ void __launch_bounds__(ATT_THREADS) decode_attn_kernel(const AttnParams p) {
    constexpr int LD = ATT_LDH(HD), KS = HD / 16, PPR = HD / 8;
    const int kvh = blockIdx.x, r = blockIdx.y, sp = blockIdx.z;
    pdl_launch_dependents();
    pdl_wait();                                  // Q, and the K/V row of this step, come from the kernels before
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int G = p.nq / p.nkv;
    const RowMeta rm = p.rows[r];
    const int extra = rm.mask ? 64 - __clzll((long long)rm.mask) : 0;
    const int total = rm.ctx + extra;
    // short contexts do not pay for a cross-CTA merge: one split per ATT_MIN_SPLIT_LEN slots
    const int nsplit = max(1, min(p.splits, (total + ATT_MIN_SPLIT_LEN - 1) / ATT_MIN_SPLIT_LEN));
    if (sp >= nsplit) return;
    const int per = (total + nsplit - 1) / nsplit;
    const int s0 = sp * per, s1 = min(total, s0 + per);

    __shared__ float sm_m[ATT_WARPS][ATT_MAX_G], sm_l[ATT_WARPS][ATT_MAX_G];
    // dynamic shared memory: [ATT_WARPS][K | V][16 slots][LD]; afterwards the merge buffer [ATT_WARPS][G][HD + 8]
    extern __shared__ __align__(16) unsigned char att_smem[];
    float* sm_acc = (float*)att_smem;
    __half* Kw = (__half*)att_smem + (size_t)warp * 2 * ATT_SLOTS * LD;
    __half* Vw = Kw + ATT_SLOTS * LD;
    __shared__ int s_last;
    __shared__ float sm_f[32][ATT_MAX_G], sm_ls[32][ATT_MAX_G], sm_linv[ATT_MAX_G];

    // A warp stages its own slots (slot = sb + row), so no barrier is involved; the K rows of its next pass are
    // requested as soon as the scores are formed, the V rows as soon as the output is.
    const size_t base = ((size_t)rm.seq * p.max_seq) * p.nkv * HD + (size_t)kvh * HD;
    const size_t stride = (size_t)p.nkv * HD;
    // 16-byte pieces where both caches start on such a boundary, else as many bytes as a lane's share of a row
    const bool wide = (((uintptr_t)p.kcache | (uintptr_t)p.vcache) & 15) == 0;
    auto copy8 = [&](__half* dst, const __half* src) {
        if (HD == 256 || wide) { cp_async16(dst, src); return; }
#pragma unroll
        for (int i = 0; i < 8; i += HD / 32) {
            if constexpr (HD == 128) cp_async8(dst + i, src + i); else cp_async4(dst + i, src + i);
        }
    };
    auto stage = [&](__half* dst, const __half* cache, int sb) {
#pragma unroll 4
        for (int i = lane; i < ATT_SLOTS * PPR; i += 32) {
            const int row = i / PPR, c = i % PPR * 8;
            if (sb + row < s1) copy8(dst + row * LD + c, cache + base + (size_t)(sb + row) * stride + c);
            else *(uint4*)(dst + row * LD + c) = make_uint4(0u, 0u, 0u, 0u);
        }
    };
    int sb = s0 + warp * ATT_SLOTS;
    stage(Kw, p.kcache, sb);
    cp_async_commit();
    stage(Vw, p.vcache, sb);
    cp_async_commit();
    // Q as B operand: head g of the group, dims 16 k + 2 t (+ 8)
    uint32_t qf[KS][2];
    {
        const __half* q = p.q + (size_t)r * p.ldq + (size_t)(kvh * G + min(g, G - 1)) * HD + 2 * t;
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            qf[k][0] = g < G ? *(const uint32_t*)(q + 16 * k) : 0u;
            qf[k][1] = g < G ? *(const uint32_t*)(q + 16 * k + 8) : 0u;
        }
    }
    const __half* ka = Kw + (lane & 15) * LD + (lane >> 4) * 8;                                  // slots x dims
    const __half* va = Vw + ((lane & 7) + (lane >> 4) * 8) * LD + ((lane >> 3) & 1) * 8;         // its transpose: dims x slots
    const float sc = p.scale * 1.44269504f;                      // scores are kept in the log2 domain
    float o[KS][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};      // o: dims 16 k + g (+ 8), heads 2 t and 2 t + 1
#pragma unroll
    for (int k = 0; k < KS; ++k) o[k][0] = o[k][1] = o[k][2] = o[k][3] = 0.f;
    for (; sb < s1; sb += ATT_MIN_SPLIT_LEN) {
        const bool more = sb + ATT_MIN_SPLIT_LEN < s1;
        cp_async_wait<1>();
        __syncwarp();
        float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < KS; k += 4) {                        // (added in pairs: short chains of roundings)
            float x[4][4] = {};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t a[4];
                at_ldsm4(a, ka + 16 * (k + i));
                at_mma(x[i], a, qf[k + i][0], qf[k + i][1]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) s[e] += (x[0][e] + x[1][e]) + (x[2][e] + x[3][e]);
        }
        __syncwarp();
        if (more) stage(Kw, p.kcache, sb + ATT_MIN_SPLIT_LEN);
        cp_async_commit();
        // slots g, g + 8 (index e >> 1) and heads 2 t, 2 t + 1 (e & 1)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int slot = sb + g + 8 * (e >> 1), d = slot - rm.ctx;
            const bool vis = slot < s1 && (d < 0 || ((rm.mask >> d) & 1ull));
            s[e] = vis ? s[e] * sc : -INFINITY;
        }
        float pw[4];
        float cor[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float mx = fmaxf(s[h], s[2 + h]);
#pragma unroll
            for (int x = 4; x < 32; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
            const float mn = fmaxf(m[h], mx), ref = mn == -INFINITY ? 0.f : mn;
            cor[h] = exp2f(m[h] - ref);                          // exp2(-inf) = 0 on the first visible slot
            m[h] = mn;
            pw[h] = exp2f(s[h] - ref) * ATT_WEIGHT;
            pw[2 + h] = exp2f(s[2 + h] - ref) * ATT_WEIGHT;
            l[h] = l[h] * cor[h] + pw[h] + pw[2 + h];
        }
        uint32_t ph[2], pl[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const __half2 hi = __floats2half2_rn(pw[2 * i], pw[2 * i + 1]);
            const float2 f = __half22float2(hi);
            const __half2 lo = __floats2half2_rn(pw[2 * i] - f.x, pw[2 * i + 1] - f.y);
            ph[i] = at_transpose(*(const uint32_t*)&hi);
            pl[i] = at_transpose(*(const uint32_t*)&lo);
        }
        cp_async_wait<1>();
        __syncwarp();
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            uint32_t v[4];
            float x[4] = {0.f, 0.f, 0.f, 0.f};
            at_ldsm4_t(v, va + 16 * k);
            at_mma(x, v, pl[0], pl[1]);
            at_mma(x, v, ph[0], ph[1]);
#pragma unroll
            for (int e = 0; e < 4; ++e) o[k][e] = fmaf(o[k][e], cor[e & 1], x[e]);
        }
        __syncwarp();
        if (more) stage(Vw, p.vcache, sb + ATT_MIN_SPLIT_LEN);
        cp_async_commit();
    }
    cp_async_wait<0>();
    __syncthreads();                             // every warp is done with its ring: the merge buffer reuses it
    // ---- merge the warps of this CTA
    constexpr int LDO = HD + 8;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int x = 4; x < 32; x <<= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], x);
        if (2 * t + h < G) {
            if (g == 0) { sm_m[warp][2 * t + h] = m[h]; sm_l[warp][2 * t + h] = l[h]; }
            float* d = sm_acc + ((size_t)warp * G + 2 * t + h) * LDO + g;
#pragma unroll
            for (int k = 0; k < KS; ++k) { d[16 * k] = o[k][h]; d[16 * k + 8] = o[k][2 + h]; }
        }
    }
    __syncthreads();
    // thread tid handles (h, d) pairs
    float* my = p.scratch + (((size_t)r * p.nkv + kvh) * p.splits + sp) * G * (HD + 4);
    const int splits_orig = p.splits;
    for (int i = tid; i < G * HD; i += ATT_THREADS) {
        int h = i / HD, d = i % HD;
        float mm = -INFINITY;
#pragma unroll
        for (int w = 0; w < ATT_WARPS; ++w) mm = fmaxf(mm, sm_m[w][h]);
        float ll = 0.f, a = 0.f;
#pragma unroll
        for (int w = 0; w < ATT_WARPS; ++w) {
            float f = (sm_m[w][h] == -INFINITY) ? 0.f : exp2f(sm_m[w][h] - mm);
            ll += sm_l[w][h] * f;
            a += sm_acc[((size_t)w * G + h) * LDO + d] * f;
        }
        if (nsplit == 1) {
            float o = ll > 0.f ? a / ll : 0.f;
            size_t col = (size_t)(kvh * G + h) * HD + d;
            if (p.gate_off >= 0) o *= sigmoid_f(__half2float(p.q[(size_t)r * p.ldq + p.gate_off + col]));
            p.out[(size_t)r * p.ldo + col] = __float2half(o);
        } else {
            my[h * (HD + 4) + d] = a;
            if (d == 0) { my[h * (HD + 4) + HD] = mm; my[h * (HD + 4) + HD + 1] = ll; }
        }
    }
    if (nsplit == 1) return;
    // ---- merge the splits: last CTA of this (row, kv head)
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        int old = atomicAdd(&p.counters[r * p.nkv + kvh], 1);
        s_last = (old == nsplit - 1);
        if (s_last) p.counters[r * p.nkv + kvh] = 0;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    const float* all = p.scratch + (((size_t)r * p.nkv + kvh) * splits_orig) * G * (HD + 4);
    // phase 1: per (split, head) rescale factors, one round trip
    for (int idx = tid; idx < nsplit * G; idx += ATT_THREADS) {
        int s = idx / G, h = idx % G;
        const float* e = &all[(size_t)(s * G + h) * (HD + 4)];
        sm_f[s][h] = ld_cg_f32(e + HD);                 // max of split s
        sm_ls[s][h] = ld_cg_f32(e + HD + 1);            // its sum
    }
    __syncthreads();
    if (tid < G) {
        float mm = -INFINITY;
        for (int s = 0; s < nsplit; ++s) mm = fmaxf(mm, sm_f[s][tid]);
        float ll = 0.f;
        for (int s = 0; s < nsplit; ++s) {
            float f = (sm_f[s][tid] == -INFINITY) ? 0.f : exp2f(sm_f[s][tid] - mm);
            ll += sm_ls[s][tid] * f;
            sm_f[s][tid] = f;
        }
        sm_linv[tid] = ll > 0.f ? 1.f / ll : 0.f;
    }
    __syncthreads();
    // phase 2: weighted sum of the partial outputs, four columns per thread; the loads of up to eight splits
    // are issued together (a loop of load-then-accumulate would wait for every load in turn)
    for (int i = tid; i < G * (HD / 4); i += ATT_THREADS) {
        const int h = i / (HD / 4), d = (i % (HD / 4)) * 4;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int sb = 0; sb < nsplit; sb += 8) {
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                v[u] = (sb + u < nsplit) ? ld_cg_v4(&all[(size_t)((sb + u) * G + h) * (HD + 4) + d]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float f = (sb + u < nsplit) ? sm_f[sb + u][h] : 0.f;
                a.x += v[u].x * f; a.y += v[u].y * f; a.z += v[u].z * f; a.w += v[u].w * f;
            }
        }
        const float li = sm_linv[h];
        const size_t col = (size_t)(kvh * G + h) * HD + d;
        float o[4] = {a.x * li, a.y * li, a.z * li, a.w * li};
        if (p.gate_off >= 0) {
            const uint2 gq = *(const uint2*)(p.q + (size_t)r * p.ldq + p.gate_off + col);
            const float2 g0 = __half22float2(*(const __half2*)&gq.x), g1 = __half22float2(*(const __half2*)&gq.y);
            o[0] *= sigmoid_f(g0.x); o[1] *= sigmoid_f(g0.y); o[2] *= sigmoid_f(g1.x); o[3] *= sigmoid_f(g1.y);
        }
        __half2 o01 = __floats2half2_rn(o[0], o[1]), o23 = __floats2half2_rn(o[2], o[3]);
        uint2 st;
        st.x = *(uint32_t*)&o01; st.y = *(uint32_t*)&o23;
        *(uint2*)(p.out + (size_t)r * p.ldo + col) = st;
    }
}

template <int HD>
static int launch_decode_attn(const AttnParams* p, cudaStream_t s) {
    dim3 grid(p->nkv, p->n_rows, p->splits);
    const size_t ring = (size_t)ATT_WARPS * 2 * ATT_SLOTS * ATT_LDH(HD) * sizeof(__half);
    const size_t merge = (size_t)ATT_WARPS * (p->nq / p->nkv) * (HD + 8) * sizeof(float);
    const size_t smem = ring > merge ? ring : merge;
    static SmemOptIn opt;
    if (int e = opt.ensure((const void*)decode_attn_kernel<HD>, smem)) return e;
    return launch_pdl(decode_attn_kernel<HD>, grid, dim3(ATT_THREADS), smem, s, *p);
}

B2_API int b2_decode_attn(const AttnParams* p, int hd, cudaStream_t s) {
    if (p->nq % p->nkv || p->nq / p->nkv > ATT_MAX_G || p->splits < 1 || p->splits > 32) return cudaErrorInvalidValue;
    if (hd == 256) return launch_decode_attn<256>(p, s);
    if (hd == 128) return launch_decode_attn<128>(p, s);
    if (hd == 64) return launch_decode_attn<64>(p, s);
    return cudaErrorInvalidValue;
}
B2_API int b2_sizeof_attn_params() { return (int)sizeof(AttnParams); }
