// Windowed attention of a decode step: split-KV flash decoding, any head size up to 256, bf16 or fp32 cache.  The work of
// one CTA, for the kernel that does this alone (csrc/attention_window.cu) and the one that runs the recurrence of a parallel
// mixer beside it (csrc/mix_decode.cu).
#pragma once
#include "mixers.cuh"

#define WD_WARPS 8
#define WD_THREADS (WD_WARPS * 32)
#define WD_GT 8                  // query heads per CTA
#define WD_KEYS 4                // keys of a warp per soft-max update (and as many on their way)
#define WD_MIN_SPLIT 64          // keys that are worth a CTA of their own
#define WD_MAX_SPLITS 32

// EPL consecutive elements of a cache row, as loaded
template <typename T, int EPL> struct WRaw { uint32_t w[EPL * sizeof(T) / 4]; };
template <typename T, int EPL>
__device__ __forceinline__ void wr_load(WRaw<T, EPL>& v, const T* p, bool ok) {
    constexpr int NW = EPL * sizeof(T) / 4;
#pragma unroll
    for (int i = 0; i < NW; ++i) v.w[i] = 0u;
    if (!ok) return;
    if constexpr (NW % 4 == 0) {
#pragma unroll
        for (int i = 0; i < NW / 4; ++i) {
            const uint4 u = ((const uint4*)p)[i];
            v.w[4 * i] = u.x; v.w[4 * i + 1] = u.y; v.w[4 * i + 2] = u.z; v.w[4 * i + 3] = u.w;
        }
    } else if constexpr (NW == 2) { const uint2 u = *(const uint2*)p; v.w[0] = u.x; v.w[1] = u.y; }
    else v.w[0] = *(const uint32_t*)p;
}
template <typename T, int EPL>
__device__ __forceinline__ float wr_get(const WRaw<T, EPL>& v, int e) {
    if constexpr (sizeof(T) == 4) return __uint_as_float(v.w[e]);
    else return __uint_as_float((e & 1) ? (v.w[e >> 1] & 0xffff0000u) : (v.w[e >> 1] << 16));
}

// The work of CTA (bx, row r, cache slice sp) of a grid (G * head blocks, rows, splits).
// EXT: kept first keys, capped scores, a sink, values of another size than the keys
template <typename T, int EPL, int GT, bool EXT>
__device__ __forceinline__ void window_decode_cta(const MixLayer& L, const MixRun& R, const int bx, const int r, const int sp) {
    const int Gq = L.H / L.G, nhb = (Gq + GT - 1) / GT;
    const int kvh = bx / nhb, hb = (bx % nhb) * GT, nh = min(GT, Gq - hb);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const RowMeta rm = R.rows[r];
    const int k1 = rm.pos + 1;                                               // keys [k0, k1)
    const int k0 = L.window > 0 ? max(0, k1 - L.window) : 0;
    // the keys a row sees, in order: kf kept first ones, then its window
    const int kf = EXT ? min(L.keep_first, k0) : 0, total = kf + k1 - k0, jump = k0 - kf;
    const int nsplit = max(1, min(R.splits, (total + WD_MIN_SPLIT - 1) / WD_MIN_SPLIT));
    if (sp >= nsplit) return;
    const int per = (total + nsplit - 1) / nsplit;
    const int a0 = sp * per, a1 = min(total, a0 + per);
    __shared__ float sm_m[WD_WARPS][GT], sm_l[WD_WARPS][GT], sm_f[WD_MAX_SPLITS][GT], sm_li[GT];
    __shared__ float sm_acc[WD_WARPS][32 * EPL];
    __shared__ int s_last;
    pdl_wait();
    const int col = lane * EPL;
    const bool in = col < L.dp, in_v = EXT ? col < L.vp : in;           // multiples of EPL (<= 8): lanes are in or out as a whole
    // Scores of WD_KEYS keys x GT heads are summed over the lanes by recursive halving: every step a lane hands
    // half of its values to its partner and keeps the other half, so afterwards each lane holds ONE finished
    // score (the value with index lane >> SH) and the soft-max costs one exponential per lane.  The running
    // maximum and sum of a head live in the lanes of its scores.
    constexpr int NV = WD_KEYS * GT, SH = NV == 32 ? 0 : NV == 16 ? 1 : NV == 8 ? 2 : 3;
    const int mykey = (lane >> SH) & (WD_KEYS - 1);
    float q[GT][EPL], acc[GT][EPL], m_l = -INFINITY, l_l = 0.f;
#pragma unroll
    for (int h = 0; h < GT; ++h) {
        WRaw<T, EPL> qv;
        wr_load(qv, (const T*)R.qbuf + ((size_t)r * L.H + kvh * Gq + hb + h) * L.dp + col, in && h < nh);
#pragma unroll
        for (int e = 0; e < EPL; ++e) { q[h][e] = wr_get(qv, e) * L.attn_scale; acc[h][e] = 0.f; }
    }
    const size_t base = (size_t)rm.seq * L.max_seq * L.G + kvh, stride = (size_t)L.G * L.dp, vstride = EXT ? (size_t)L.G * L.vp : stride;
    const T* kc = (const T*)L.kcache + base * L.dp + col;
    const T* vc = (const T*)L.vcache + base * (EXT ? L.vp : L.dp) + col;
    const int dv = EXT ? L.dv : L.d;
    WRaw<T, EPL> kn[WD_KEYS], vn[WD_KEYS];
    auto fetch = [&](int s) {
#pragma unroll
        for (int i = 0; i < WD_KEYS; ++i) {
            const int idx = s + i * WD_WARPS + warp, key = EXT && idx < kf ? idx : idx + jump;
            const bool ok = idx < a1;
            wr_load(kn[i], kc + (size_t)key * stride, in && ok);
            wr_load(vn[i], vc + (size_t)key * vstride, in_v && ok);
        }
    };
    if (a0 < a1) fetch(a0);
    for (int s = a0; s + warp < a1; s += WD_WARPS * WD_KEYS) {
        WRaw<T, EPL> kk[WD_KEYS], vv[WD_KEYS];
#pragma unroll
        for (int i = 0; i < WD_KEYS; ++i) { kk[i] = kn[i]; vv[i] = vn[i]; }
        if (s + WD_WARPS * WD_KEYS < a1) fetch(s + WD_WARPS * WD_KEYS);
        float d[NV];                                         // [head][key]
#pragma unroll
        for (int h = 0; h < GT; ++h)
#pragma unroll
            for (int i = 0; i < WD_KEYS; ++i) {
                float x = 0.f;
                if (h < nh)
#pragma unroll
                    for (int e = 0; e < EPL; ++e) x = fmaf(q[h][e], wr_get(kk[i], e), x);
                d[h * WD_KEYS + i] = x;
            }
        int off = 16;
#pragma unroll
        for (int n = NV; n > 1; n >>= 1, off >>= 1) {
            const bool up = lane & off;
#pragma unroll
            for (int i = 0; i < n / 2; ++i) {
                const float give = up ? d[i] : d[i + n / 2], keep = up ? d[i + n / 2] : d[i];
                d[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
            }
        }
#pragma unroll
        for (int o = 16 / NV; o > 0; o >>= 1) d[0] += __shfl_xor_sync(0xffffffffu, d[0], o);
        if (EXT && L.softcap > 0.f) d[0] = L.softcap * tanhf(d[0] / L.softcap);
        const float sc = s + mykey * WD_WARPS + warp < a1 ? d[0] : -INFINITY;
        float mn = sc;
#pragma unroll
        for (int o = 1; o < WD_KEYS; o <<= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, o << SH));
        mn = fmaxf(mn, m_l);                                 // (the first key of the pass is always inside: finite)
        const float corr_l = expf(m_l - mn), p_l = expf(sc - mn);
        float ps = p_l;
#pragma unroll
        for (int o = 1; o < WD_KEYS; o <<= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o << SH);
        l_l = l_l * corr_l + ps;
        m_l = mn;
#pragma unroll
        for (int h = 0; h < GT; ++h) {
            if (h >= nh) break;
            const float corr = __shfl_sync(0xffffffffu, corr_l, (h * WD_KEYS) << SH);
            float pw[WD_KEYS];
#pragma unroll
            for (int i = 0; i < WD_KEYS; ++i) pw[i] = __shfl_sync(0xffffffffu, p_l, (h * WD_KEYS + i) << SH);
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
                float a = acc[h][e] * corr;
#pragma unroll
                for (int i = 0; i < WD_KEYS; ++i) a = fmaf(pw[i], wr_get(vv[i], e), a);
                acc[h][e] = a;
            }
        }
    }
    // ---- merge the warps, one head at a time
    if ((lane & ((WD_KEYS << SH) - 1)) == 0) { sm_m[warp][lane / (WD_KEYS << SH)] = m_l; sm_l[warp][lane / (WD_KEYS << SH)] = l_l; }
    const int unit = (r * L.G + kvh) * nhb + bx % nhb;
    float* my = R.attn_scratch + ((size_t)unit * R.splits + sp) * GT * (32 * EPL + 4);
#pragma unroll
    for (int h = 0; h < GT; ++h) {
        if (h >= nh) break;
        __syncthreads();
#pragma unroll
        for (int e = 0; e < EPL; ++e) sm_acc[warp][col + e] = acc[h][e];
        __syncthreads();
        float mm = -INFINITY;
#pragma unroll
        for (int w = 0; w < WD_WARPS; ++w) mm = fmaxf(mm, sm_m[w][h]);
        const int head = kvh * Gq + hb + h;
        const bool sink = EXT && L.sink && nsplit == 1;             // (slices: the merge below counts it)
        if (sink) mm = fmaxf(mm, L.sink[head]);
        float ll = sink ? expf(L.sink[head] - mm) : 0.f, f[WD_WARPS];
#pragma unroll
        for (int w = 0; w < WD_WARPS; ++w) { f[w] = sm_m[w][h] == -INFINITY ? 0.f : expf(sm_m[w][h] - mm); ll += sm_l[w][h] * f[w]; }
        for (int c = tid; c < dv; c += WD_THREADS) {
            float a = 0.f;
#pragma unroll
            for (int w = 0; w < WD_WARPS; ++w) a += sm_acc[w][c] * f[w];
            if (nsplit == 1) ((T*)R.out)[(size_t)r * R.ldo + head * dv + c] = to_t<T>(a / ll * L.left_scale);
            else {
                my[h * (32 * EPL + 4) + c] = a;
                if (c == 0) { my[h * (32 * EPL + 4) + 32 * EPL] = mm; my[h * (32 * EPL + 4) + 32 * EPL + 1] = ll; }
            }
        }
    }
    if (nsplit == 1) return;
    // ---- merge the slices: the last CTA of this (row, key head, head block)
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const int old = atomicAdd(&R.attn_counters[unit], 1);
        s_last = old == nsplit - 1;
        if (s_last) R.attn_counters[unit] = 0;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    const float* all = R.attn_scratch + (size_t)unit * R.splits * GT * (32 * EPL + 4);
    if (tid < nh) {
        const float* e0 = all + tid * (32 * EPL + 4) + 32 * EPL;
        const size_t st = (size_t)GT * (32 * EPL + 4);
        float mv[WD_MAX_SPLITS], lv[WD_MAX_SPLITS], mm = -INFINITY, ll = 0.f;
#pragma unroll
        for (int x = 0; x < WD_MAX_SPLITS; ++x) {
            mv[x] = x < nsplit ? __ldcg(e0 + x * st) : -INFINITY;
            lv[x] = x < nsplit ? __ldcg(e0 + x * st + 1) : 0.f;
        }
#pragma unroll
        for (int x = 0; x < WD_MAX_SPLITS; ++x) mm = fmaxf(mm, mv[x]);
        if (EXT && L.sink) { const float sk = L.sink[kvh * Gq + hb + tid]; mm = fmaxf(mm, sk); ll = expf(sk - mm); }
#pragma unroll
        for (int x = 0; x < WD_MAX_SPLITS; ++x) {
            const float f = mv[x] == -INFINITY ? 0.f : expf(mv[x] - mm);
            ll += lv[x] * f;
            sm_f[x][tid] = f;
        }
        sm_li[tid] = 1.f / ll;
    }
    __syncthreads();
    for (int i = tid; i < nh * dv; i += WD_THREADS) {
        const int h = i / dv, c = i % dv;
        float a = 0.f;
        for (int x0 = 0; x0 < nsplit; x0 += 8) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                v[u] = x0 + u < nsplit ? __ldcg(all + ((size_t)(x0 + u) * GT + h) * (32 * EPL + 4) + c) : 0.f;
#pragma unroll
            for (int u = 0; u < 8; ++u) if (x0 + u < nsplit) a = fmaf(v[u], sm_f[x0 + u][h], a);
        }
        ((T*)R.out)[(size_t)r * R.ldo + (kvh * Gq + hb + h) * dv + c] = to_t<T>(a * sm_li[h] * L.left_scale);
    }
}

// Cache slices of a launch with this many CTAs resident at once: more would only add a second wave.
static inline int window_decode_splits(const MixLayer* l, const MixRun* r, int slots) {
    const int units = l->G * ((l->H / l->G + WD_GT - 1) / WD_GT) * r->n_rows;
    return units * r->splits > slots ? (units >= slots ? 1 : slots / units) : r->splits;
}
