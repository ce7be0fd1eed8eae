// Sliding-window attention, and the preparation pass in front of a mixer.
//
//   mix_prepare       parallel mixer: RMSNorm of Q and of K over the WHOLE projection (all heads at once), rotation
//                     of the first `rot` dimensions of every head in (i, i + rot/2) pairs, K and the values into the
//                     cache, causal convolution + SiLU of the recurrence's inputs, its step sizes.
//   head_prepare      attention alone: RMSNorm of every Q and K head with one weight for all heads, optional
//                     rotation, K and the values into the cache.
//   window decode     split-KV flash decoding, any head size up to 256, bf16 or fp32 cache.
//   (many query rows of one sequence: csrc/attention_window_rows.cu)
//
// Visibility: the row at position p sees slots max(0, p - window + 1) .. p of its sequence and its first
// keep_first slots (slot = position: rows of a sequence are consecutive tokens, no draft trees).  Scores may be
// capped (softcap * tanh(score / softcap)), and a learned sink per head may join the soft-max's denominator: it
// is neither scaled nor capped and has no value.
#include "mixers.cuh"
#include "window_decode.cuh"

// ---------------------------------------------------------------------------
// prepare: one-dimensional grid.  First (q_slices + 1) CTAs per row: slices of the query heads, then the keys;
// every one of them sums the squares of its whole projection.  Then the convolution: column blocks of 512
// channels times tiles of conv_rows rows.
// ---------------------------------------------------------------------------
#define MP_THREADS 256
#define MP_COLS (2 * MP_THREADS)
#define MP_MAX_ROWS 8            // rows of a convolution tile
#define MP_TAPS 4                // taps whose weights stay in registers

template <typename T>
__device__ __forceinline__ void mp_heads(const MixLayer& L, const MixRun& R, int r, int slice, int q_slices, float* sv, float* red) {
    const int tid = threadIdx.x;
    const bool is_q = slice < q_slices;
    const RowMeta rm = R.rows[r];
    const int heads = is_q ? L.H : L.G, n = heads * L.d, off = is_q ? L.off_q : L.off_k;
    const int per = is_q ? (heads + q_slices - 1) / q_slices : heads;
    const int h0 = is_q ? slice * per : 0, h1 = min(heads, h0 + per), i0 = h0 * L.d, i1 = h1 * L.d;
    const T* src = (const T*)R.proj + (size_t)r * R.ld_proj + off;
    const float* nw = is_q ? L.q_norm : L.k_norm;
    const size_t slot = ((size_t)rm.seq * L.max_seq + rm.slot) * L.G * L.dp;
    T* dst = is_q ? (T*)R.qbuf + (size_t)r * L.H * L.dp : (T*)L.kcache + slot;
    T* vdst = (T*)L.vcache + slot;                         // (values = keys as projected: vp == dp)
    constexpr int V = 16 / sizeof(T);
    const bool vec = ((off | R.ld_proj | n) & (V - 1)) == 0;
    pdl_wait();
    float ss = 0.f;
    if (vec) {
#pragma unroll 2
        for (int i = tid * V; i < n; i += MP_THREADS * V) {
            const uint4 u = *(const uint4*)(src + i);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
            float v[V];
#pragma unroll
            for (int e = 0; e < V; ++e) {
                v[e] = sizeof(T) == 4 ? __uint_as_float(w[e & 3])
                                      : __uint_as_float((e & 1) ? (w[(e >> 1) & 3] & 0xffff0000u) : (w[(e >> 1) & 3] << 16));
                ss += v[e] * v[e];
            }
            if ((i0 & 3) == 0 && i >= i0 && i + V <= i1) {
#pragma unroll
                for (int e = 0; e < V; e += 4) *(float4*)(sv + i - i0 + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
            } else
#pragma unroll
                for (int e = 0; e < V; ++e) if (i + e >= i0 && i + e < i1) sv[i + e - i0] = v[e];
        }
    } else
        for (int i = tid; i < n; i += MP_THREADS) {
            const float v = ld_f(src + i);
            ss += v * v;
            if (i >= i0 && i < i1) sv[i - i0] = v;
        }
    const float inv = rsqrtf(block_sum(ss, red) / (float)n + L.eps);      // (its barriers also publish sv)
    const int half = L.rot >> 1;
    const float* ct = L.cos_tab + (size_t)rm.pos * half;
    const float* st = L.sin_tab + (size_t)rm.pos * half;
    // Eight elements at a time where heads, their rotated halves and addresses allow it (one by one the loads of weights and angles, a
    // division and 2-byte stores for each element cost more than its bytes: 1000 rows of 40 + 8 heads of 128 and 7168 channels 59 -> 46 us
    // with the convolution's inputs requested at once and conflict-free stores)
    if (L.dp == L.d && ((L.d | half) & 7) == 0 && (((uintptr_t)nw | (uintptr_t)L.cos_tab | (uintptr_t)L.sin_tab | (uintptr_t)dst | (uintptr_t)vdst) & 15) == 0) {
        const int d8 = L.d >> 3;
        auto ld8 = [](const float* p, float (&v)[8]) {
            const float4 a = ((const float4*)p)[0], b = ((const float4*)p)[1];
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        };
        auto st8 = [](T* p, const float (&v)[8]) {
            T raw[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) raw[e] = to_t<T>(v[e]);
#pragma unroll
            for (int q = 0; q < (int)(8 * sizeof(T) / 16); ++q) ((uint4*)p)[q] = ((const uint4*)raw)[q];
        };
        for (int i = tid; i < (h1 - h0) * d8; i += MP_THREADS) {
            const int hd = i / d8, e0 = (i - hd * d8) * 8, j = hd * L.d + e0;
            float raw[8], w[8], o[8];
            ld8(sv + j, raw);
            ld8(nw + i0 + j, w);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = raw[e] * inv * w[e];
            if (e0 < L.rot) {
                const bool first = e0 < half;
                const int a = first ? e0 : e0 - half, jo = first ? j + half : j - half;
                float x[8], c[8], s[8];
                ld8(sv + jo, x);
                ld8(nw + i0 + jo, w);
                ld8(ct + a, c);
                ld8(st + a, s);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float other = x[e] * inv * w[e];
                    o[e] = first ? o[e] * c[e] - other * s[e] : o[e] * c[e] + other * s[e];
                }
            }
            st8(dst + h0 * L.dp + hd * L.dp + e0, o);
            if (!is_q) st8(vdst + hd * L.dp + e0, raw);
        }
        return;
    }
#pragma unroll 2
    for (int i = tid; i < (h1 - h0) * L.dp; i += MP_THREADS) {
        const int hd = i / L.dp, e = i - hd * L.dp, j = hd * L.d + e;
        float o = 0.f, raw = 0.f;
        if (e < L.d) {
            raw = sv[j];
            o = raw * inv * nw[i0 + j];
            if (e < L.rot) {
                const bool first = e < half;
                const int a = first ? e : e - half, jo = first ? j + half : j - half;
                const float other = sv[jo] * inv * nw[i0 + jo];
                o = first ? o * ct[a] - other * st[a] : o * ct[a] + other * st[a];
            }
        }
        dst[h0 * L.dp + i] = to_t<T>(o);
        if (!is_q) vdst[i] = to_t<T>(raw);
    }
}

// two adjacent elements (one 2 x sizeof(T) load when `pair`: the address is aligned to it)
template <typename T>
__device__ __forceinline__ float2 mp_ld2(const T* p, bool pair, bool second) {
    if (pair) {
        if constexpr (sizeof(T) == 4) return *(const float2*)p;
        else return __bfloat1622float2(*(const __nv_bfloat162*)p);
    }
    return make_float2(ld_f(p), second ? ld_f(p + 1) : 0.f);
}

template <typename T>
__device__ __forceinline__ void mp_conv(const MixLayer& L, const MixRun& R, int blk, int r0, int rows) {
    __shared__ int s_local[MP_MAX_ROWS], s_seq[MP_MAX_ROWS];
    const int tid = threadIdx.x, C = L.heads * L.P + 2 * L.groups * L.N, c = blk * MP_COLS + 2 * tid, K = L.taps - 1;
    if (tid < rows) {
        // rows of the same sequence in front of this one in the launch, as far as the taps reach
        const int r = r0 + tid, seq = R.rows[r].seq;
        int before[MP_TAPS - 1], local = 0;                  // (requested together)
#pragma unroll
        for (int j = 0; j < MP_TAPS - 1; ++j) before[j] = j < K && r - j - 1 >= 0 ? R.rows[r - j - 1].seq : -1;
#pragma unroll
        for (int j = 0; j < MP_TAPS - 1; ++j) if (local == j && j < K && before[j] == seq) ++local;
        if (local == MP_TAPS - 1) while (local < K && r - local - 1 >= 0 && R.rows[r - local - 1].seq == seq) ++local;
        s_local[tid] = local; s_seq[tid] = seq;
    }
    const bool in = c < C, second = c + 1 < C;
    const bool pair = second && ((L.off_x | R.ld_proj | C) & 1) == 0, pair_out = second && (R.ld_xbc & 1) == 0;
    float b0 = 0.f, b1 = 0.f, w0[MP_TAPS], w1[MP_TAPS];
    const bool regs = L.taps <= MP_TAPS;
    const int lead = MP_TAPS - L.taps;                      // (weights at the end of the registers: the last is the row's own)
    if (in) {
        b0 = L.conv_b[c]; b1 = second ? L.conv_b[c + 1] : 0.f;
#pragma unroll
        for (int j = 0; j < MP_TAPS; ++j) {
            w0[j] = (regs && j >= lead) ? L.conv_w[(size_t)c * L.taps + j - lead] : 0.f;
            w1[j] = (regs && j >= lead && second) ? L.conv_w[(size_t)(c + 1) * L.taps + j - lead] : 0.f;
        }
    }
    pdl_wait();
    __syncthreads();
    if (blk == 0)
        for (int i = tid; i < rows * L.heads; i += MP_THREADS) {
            const int r = r0 + i / L.heads, h = i % L.heads;
            R.dtb[(size_t)r * R.ld_dt + h] = softplus_p(ld_f((const T*)R.proj + (size_t)r * R.ld_proj + L.off_dt + h) + L.dt_bias[h]);
        }
    if (!in) return;
    auto put = [&](int r, float a0, float a1) {
        T* out = (T*)R.xbc + (size_t)r * R.ld_xbc + c;
        const T o0 = to_t<T>(silu_p(a0)), o1 = to_t<T>(silu_p(a1));
        if (pair_out) {
            if constexpr (sizeof(T) == 4) *(float2*)out = make_float2(o0, o1);
            else { __nv_bfloat162 h; h.x = o0; h.y = o1; *(__nv_bfloat162*)out = h; }
        } else { out[0] = o0; if (second) out[1] = o1; }
    };
    // the input `back` tokens before row r of a sequence with `local` rows in front of it in this launch
    auto input = [&](int r, int seq, int local, int back) {
        return back <= local ? mp_ld2((const T*)R.proj + (size_t)(r - back) * R.ld_proj + L.off_x + c, pair, second)
                             : mp_ld2((const T*)L.conv_state + ((size_t)seq * K + K - (back - local)) * C + c, pair, second);
    };
    bool same = rows > 1;                                   // (a single row needs no tile: decode at width 2048 2.30 us, as one 2.40)
    if (same)
#pragma unroll
        for (int i = 1; i < MP_MAX_ROWS; ++i) same = same && (i >= rows || s_seq[i] == s_seq[0]);
    if (regs && same) {
        // one sequence: every input of the tile is read once, all of them at once (row by row they were a trip to L2 each)
        float2 v[MP_MAX_ROWS + MP_TAPS - 1];
#pragma unroll
        for (int i = 0; i < MP_MAX_ROWS + MP_TAPS - 1; ++i) {
            const int at = i - (MP_TAPS - 1);               // relative to r0
            v[i] = at >= -K && at < rows ? (at >= 0 ? input(r0 + at, s_seq[0], 0, 0) : input(r0, s_seq[0], s_local[0], -at)) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < MP_MAX_ROWS; ++i) {
            if (i >= rows) break;
            float a0 = b0, a1 = b1;
            // (with fewer taps the first places hold inputs that this row does not see: an infinity there times a weight of zero is NaN)
#pragma unroll
            for (int j = 0; j < MP_TAPS; ++j) if (j >= lead) { a0 = fmaf(w0[j], v[i + j].x, a0); a1 = fmaf(w1[j], v[i + j].y, a1); }
            put(r0 + i, a0, a1);
        }
        return;
    }
    for (int i = 0; i < rows; ++i) {
        const int r = r0 + i, local = s_local[i], seq = s_seq[i];
        float a0 = b0, a1 = b1;
        if (regs) {
            float2 v[MP_TAPS];
#pragma unroll
            for (int j = 0; j < MP_TAPS; ++j) v[j] = j >= lead ? input(r, seq, local, MP_TAPS - 1 - j) : make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < MP_TAPS; ++j) { a0 = fmaf(w0[j], v[j].x, a0); a1 = fmaf(w1[j], v[j].y, a1); }
        } else
            for (int j = 0; j < L.taps; ++j) {
                const float2 v = input(r, seq, local, K - j);
                a0 = fmaf(L.conv_w[(size_t)c * L.taps + j], v.x, a0);
                if (second) a1 = fmaf(L.conv_w[(size_t)(c + 1) * L.taps + j], v.y, a1);
            }
        put(r, a0, a1);
    }
}

template <typename T>
__global__ void __launch_bounds__(MP_THREADS) mix_prepare_kernel(const MixLayer L, const MixRun R, int q_slices, int col_blocks, int conv_rows) {
    extern __shared__ __align__(16) float mp_v[];            // the heads a CTA rotates
    __shared__ float red[32];
    pdl_launch_dependents();
    const int nh = R.n_rows * (q_slices + 1);
    int b = blockIdx.x;
    if (b < nh) { mp_heads<T>(L, R, b / (q_slices + 1), b % (q_slices + 1), q_slices, mp_v, red); return; }
    b -= nh;
    const int r0 = (b / col_blocks) * conv_rows;
    mp_conv<T>(L, R, b % col_blocks, r0, min(conv_rows, R.n_rows - r0));
}

// ---------------------------------------------------------------------------
// head_prepare: one warp per (row, query head | key head | value head)
// ---------------------------------------------------------------------------
template <typename T, int EPL>
__global__ void __launch_bounds__(256) head_prepare_kernel(const MixLayer L, const MixRun R) {
    __shared__ float sv[8][32 * EPL];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per = L.H + L.G + (L.off_v >= 0 ? L.G : 0), unit = blockIdx.x * 8 + warp;
    if (unit >= R.n_rows * per) return;
    const int r = unit / per, j = unit % per;
    const RowMeta rm = R.rows[r];
    const bool is_q = j < L.H, is_v = j >= L.H + L.G;
    const int hd = is_q ? j : (is_v ? j - L.H - L.G : j - L.H), n = is_v ? L.dv : L.d, np = is_v ? L.vp : L.dp;
    const int off = (is_q ? L.off_q : (is_v ? L.off_v : L.off_k)) + hd * n, c0 = lane * EPL;
    const T* src = (const T*)R.proj + (size_t)r * R.ld_proj + off + c0;
    const size_t slot = ((size_t)rm.seq * L.max_seq + rm.slot) * L.G + hd;
    T* dst = is_q ? (T*)R.qbuf + ((size_t)r * L.H + hd) * L.dp : (is_v ? (T*)L.vcache + slot * L.vp : (T*)L.kcache + slot * L.dp);
    const float* nw = is_q ? L.q_norm : L.k_norm;
    const bool vec = ((off | n | R.ld_proj) & (EPL - 1)) == 0;
    float w[EPL], v[EPL], ss = 0.f;
#pragma unroll
    for (int e = 0; e < EPL; ++e) w[e] = (!is_v && c0 + e < n) ? nw[c0 + e] : 0.f;
    pdl_wait();
#pragma unroll
    for (int e = 0; e < EPL; ++e) v[e] = 0.f;
    if (vec && c0 < n) {
        T raw[EPL];
        if constexpr (EPL * sizeof(T) == 4) *(uint32_t*)raw = *(const uint32_t*)src;
        else if constexpr (EPL * sizeof(T) == 8) *(uint2*)raw = *(const uint2*)src;
        else
#pragma unroll
            for (int i = 0; i < (int)(EPL * sizeof(T) / 16); ++i) ((uint4*)raw)[i] = ((const uint4*)src)[i];
#pragma unroll
        for (int e = 0; e < EPL; ++e) v[e] = ld_f(raw + e);
    } else
#pragma unroll
        for (int e = 0; e < EPL; ++e) if (c0 + e < n) v[e] = ld_f(src + e);
    auto put = [&](T* d, int len, const float (&o)[EPL]) {          // (len is a multiple of 8)
        if (c0 >= len) return;
        T raw[EPL];
#pragma unroll
        for (int e = 0; e < EPL; ++e) raw[e] = to_t<T>(o[e]);
        if constexpr (EPL * sizeof(T) == 4) *(uint32_t*)(d + c0) = *(const uint32_t*)raw;
        else if constexpr (EPL * sizeof(T) == 8) *(uint2*)(d + c0) = *(const uint2*)raw;
        else
#pragma unroll
            for (int i = 0; i < (int)(EPL * sizeof(T) / 16); ++i) ((uint4*)(d + c0))[i] = ((const uint4*)raw)[i];
    };
    if (is_v) { put(dst, np, v); return; }
    if (!is_q && L.off_v < 0) put((T*)L.vcache + slot * L.vp, L.vp, v);
#pragma unroll
    for (int e = 0; e < EPL; ++e) ss += v[e] * v[e];
    const float inv = rsqrtf(warp_sum(ss) / (float)n + L.eps);
#pragma unroll
    for (int e = 0; e < EPL; ++e) v[e] *= inv * w[e];
    if (L.rot > 0) {
        const int half = L.rot >> 1;
        const float* ct = L.cos_tab + (size_t)rm.pos * half;
        const float* st = L.sin_tab + (size_t)rm.pos * half;
#pragma unroll
        for (int e = 0; e < EPL; ++e) sv[warp][c0 + e] = v[e];
        __syncwarp();
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
            const int i = c0 + e;
            if (i >= L.rot) continue;
            const bool first = i < half;
            const int a = first ? i : i - half;
            const float other = sv[warp][first ? i + half : a];
            v[e] = first ? v[e] * ct[a] - other * st[a] : v[e] * ct[a] + other * st[a];
        }
    }
    put(dst, np, v);
}
template <typename T>
static int launch_hp(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    const int per = l->H + l->G + (l->off_v >= 0 ? l->G : 0), m = l->dp > l->vp ? l->dp : l->vp;
    const dim3 grid((r->n_rows * per + 7) / 8), block(256);
    if (m <= 64) return launch_pdl(head_prepare_kernel<T, 2>, grid, block, 0, s, *l, *r);
    if (m <= 128) return launch_pdl(head_prepare_kernel<T, 4>, grid, block, 0, s, *l, *r);
    return launch_pdl(head_prepare_kernel<T, 8>, grid, block, 0, s, *l, *r);
}

B2_API int b2_head_prepare(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    if (!attn_valid(l) || !l->head_norm || !l->q_norm || !l->k_norm || (l->off_v < 0 && l->dv != l->d) || (l->rot > 0 && !l->cos_tab))
        return cudaErrorInvalidValue;
    return r->dt == DT_BF16 ? launch_hp<bf16>(l, r, s) : launch_hp<float>(l, r, s);
}

B2_API int b2_mix_prepare(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    if (!attn_valid(l) || l->head_norm || l->off_v >= 0 || l->dv != l->d) return cudaErrorInvalidValue;
    if (l->H < 1 || l->G < 1 || l->H % l->G || l->d > 256 || l->dp < l->d || (l->dp & 7) || l->rot > l->d || (l->rot & 1) ||
        l->taps < 1 || l->groups < 1 || l->heads % l->groups)
        return cudaErrorInvalidValue;
    const int C = l->heads * l->P + 2 * l->groups * l->N;
    // few rows: cut the query heads so that a slice is one pass of a CTA; many rows fill the GPU as they are
    int qs = r->n_rows <= B2_MAX_ROWS ? (l->H * l->d + 511) / 512 : 1;
    if (qs > l->H) qs = l->H;
    const int per = (l->H + qs - 1) / qs;
    qs = (l->H + per - 1) / per;
    const int cb = (C + MP_COLS - 1) / MP_COLS, cr = r->n_rows <= B2_MAX_ROWS ? 1 : MP_MAX_ROWS;
    const dim3 grid(r->n_rows * (qs + 1) + cb * ((r->n_rows + cr - 1) / cr));
    const size_t smem = (size_t)(per > l->G ? per : l->G) * l->d * sizeof(float);
    static SmemOptIn opt[2];
    if (r->dt == DT_BF16) {
        if (int e = opt[0].ensure((const void*)mix_prepare_kernel<bf16>, smem)) return e;
        return launch_pdl(mix_prepare_kernel<bf16>, grid, dim3(MP_THREADS), smem, s, *l, *r, qs, cb, cr);
    }
    if (int e = opt[1].ensure((const void*)mix_prepare_kernel<float>, smem)) return e;
    return launch_pdl(mix_prepare_kernel<float>, grid, dim3(MP_THREADS), smem, s, *l, *r, qs, cb, cr);
}

// ---------------------------------------------------------------------------
// decode: grid (G * head blocks, rows, splits)
// ---------------------------------------------------------------------------
template <typename T, int EPL, int GT, bool EXT>
__global__ void __launch_bounds__(WD_THREADS) window_decode_kernel(const MixLayer L, const MixRun R) {
    pdl_launch_dependents();
    window_decode_cta<T, EPL, GT, EXT>(L, R, blockIdx.x, blockIdx.y, blockIdx.z);
}

// floats of scratch for `rows` rows, dp: the larger of MixLayer's dp and vp (attn_counters: rows * G * ceil(H / G / WD_GT) ints)
B2_API long long b2_window_attn_scratch(int H, int G, int dp, int rows, int splits) {
    const int nhb = (H / G + WD_GT - 1) / WD_GT, epl = dp <= 64 ? 2 : dp <= 128 ? 4 : 8;
    return (long long)rows * G * nhb * splits * WD_GT * (32 * epl + 4);
}
B2_API int b2_window_attn_units(int H, int G, int rows) { return rows * G * ((H / G + WD_GT - 1) / WD_GT); }

template <typename T, int EPL, bool EXT>
static int launch_wd(const MixLayer* l, const MixRun* run, cudaStream_t s) {
    const int Gq = l->H / l->G;
    // cache slices beyond what is resident at once would only add a second wave
    MixRun one = *run;
    one.splits = window_decode_splits(l, run, 148 * (Gq > 4 || EPL > 4 ? 1 : 2));
    const MixRun* r = &one;
    // (a smaller head block keeps fewer registers; scratch is laid out for at most WD_GT heads per block)
    if (Gq <= 1) return launch_pdl(window_decode_kernel<T, EPL, 1, EXT>, dim3(l->G, r->n_rows, r->splits), dim3(WD_THREADS), 0, s, *l, *r);
    if (Gq <= 2) return launch_pdl(window_decode_kernel<T, EPL, 2, EXT>, dim3(l->G, r->n_rows, r->splits), dim3(WD_THREADS), 0, s, *l, *r);
    if (Gq <= 4) return launch_pdl(window_decode_kernel<T, EPL, 4, EXT>, dim3(l->G, r->n_rows, r->splits), dim3(WD_THREADS), 0, s, *l, *r);
    const int nhb = (Gq + WD_GT - 1) / WD_GT;
    return launch_pdl(window_decode_kernel<T, EPL, WD_GT, EXT>, dim3(l->G * nhb, r->n_rows, r->splits), dim3(WD_THREADS), 0, s, *l, *r);
}
template <typename T, bool EXT>
static int launch_wd_t(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    const int m = l->dp > l->vp ? l->dp : l->vp;
    if (m <= 64) return launch_wd<T, 2, EXT>(l, r, s);
    if (m <= 128) return launch_wd<T, 4, EXT>(l, r, s);
    return launch_wd<T, 8, EXT>(l, r, s);
}
B2_API int b2_window_attn_decode(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    if (!attn_valid(l) || r->splits < 1 || r->splits > WD_MAX_SPLITS) return cudaErrorInvalidValue;
    const bool ext = l->keep_first > 0 || l->softcap > 0.f || l->sink || l->dv != l->d;
    if (r->dt == DT_BF16) return ext ? launch_wd_t<bf16, true>(l, r, s) : launch_wd_t<bf16, false>(l, r, s);
    return ext ? launch_wd_t<float, true>(l, r, s) : launch_wd_t<float, false>(l, r, s);
}

B2_API int b2_sizeof_mix_layer() { return (int)sizeof(MixLayer); }
B2_API int b2_sizeof_mix_run() { return (int)sizeof(MixRun); }
