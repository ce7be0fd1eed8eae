// A linear recurrence token by token: the work of one CTA (head, 32 columns of P, sequence), for the kernel that does this
// alone (csrc/ssd.cu) and the one that runs the attention of a parallel mixer beside it (csrc/mix_decode.cu).
// lane = column of P, warp = slice of N; the state in registers.
#pragma once
#include "mixers.cuh"

// The last taps-1 raw inputs of the channels [c0, c1) after this launch's rows [r0, r1) of one sequence.
// Ascending in place: entry i takes the old entry i + n (n rows) or a row of the projection.
template <typename T>
__device__ __forceinline__ void conv_history(const MixLayer& L, const MixRun& R, int seq, int r0, int r1, int c0, int c1,
                                             int tid, int nthr) {
    const int C = L.heads * L.P + 2 * L.groups * L.N, K = L.taps - 1, n = r1 - r0;
    if (K == 0) return;
    T* hist = (T*)L.conv_state + (size_t)seq * K * C;
    for (int c = c0 + tid; c < c1; c += nthr)
        for (int i = 0; i < K; ++i) {
            const int back = n - K + i;                     // row index of the input that lands in entry i
            hist[(size_t)i * C + c] = back >= 0 ? ((const T*)R.proj)[(size_t)(r0 + back) * R.ld_proj + L.off_x + c]
                                                : hist[(size_t)(i + n) * C + c];
        }
}
// Channels a CTA (head h, column block of width pw at p0) carries over: its own x columns, and for the
// first head of a group and the first block also the group's B and C.
template <typename T>
__device__ __forceinline__ void conv_history_of(const MixLayer& L, const MixRun& R, int seq, int r0, int r1, int h, int p0, int pw,
                                                int tid, int nthr) {
    const int I = L.heads * L.P, rep = L.heads / L.groups;
    conv_history<T>(L, R, seq, r0, r1, h * L.P + p0, h * L.P + min(L.P, p0 + pw), tid, nthr);
    if (p0 == 0 && h % rep == 0) {
        const int g = h / rep;
        conv_history<T>(L, R, seq, r0, r1, I + g * L.N, I + (g + 1) * L.N, tid, nthr);
        conv_history<T>(L, R, seq, r0, r1, I + (L.groups + g) * L.N, I + (L.groups + g + 1) * L.N, tid, nthr);
    }
}

__device__ __forceinline__ uint32_t sc_pack(bf16 a, bf16 b) {
    return (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
}
// log decay and step size of the token in row r
__device__ __forceinline__ float rec_rate(const MixLayer& L, int h) { return L.decay ? L.log_decay[h] : -expf(L.A_log[h]); }
__device__ __forceinline__ float rec_dt(const MixLayer& L, const MixRun& R, int r, int h) {
    return L.decay ? 1.f : R.dtb[(size_t)r * R.ld_dt + h];
}

// RMSNorm of one part of one row: out = u / rms(u) * w * right_scale (* sigmoid(z)), from column out_col on.
#define NP_REGS 4                // float4s per thread that stay in registers between the passes
template <typename T>
__device__ __forceinline__ void norm_part(const MixLayer& L, const MixRun& R, int r, int part, float* red) {
    const int I = L.heads * L.P, w = I / L.ngroups, c0 = part * w, tid = threadIdx.x, nt = blockDim.x;
    const float* u = R.ubuf + (size_t)r * R.ld_u + c0;
    const float* nw = L.norm_w + c0;
    T* out = (T*)R.out + (size_t)r * R.ldo + L.out_col + c0;
    const T* z = (const T*)R.proj + (size_t)r * R.ld_proj + L.off_z + c0;
    const bool gate = L.gate == REC_NORM_SIGMOID;
    auto one = [&](int i, float v, float inv) {
        v *= inv * nw[i] * L.right_scale;
        out[i] = to_t<T>(gate ? v * sigmoid_p(ld_f(z + i)) : v);
    };
    float ss = 0.f;
    if (((w | c0 | R.ld_u) & 3) == 0) {
        float4 v[NP_REGS];
        const int w4 = w >> 2;
#pragma unroll
        for (int j = 0; j < NP_REGS; ++j) {
            const int i = tid + j * nt;
            v[j] = i < w4 ? __ldcg((const float4*)u + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < NP_REGS; ++j) ss += v[j].x * v[j].x + v[j].y * v[j].y + v[j].z * v[j].z + v[j].w * v[j].w;
        for (int i = tid + NP_REGS * nt; i < w4; i += nt) {
            const float4 q = __ldcg((const float4*)u + i);
            ss += q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w;
        }
        const float inv = rsqrtf(block_sum(ss, red) / (float)w + L.eps);
        const bool packed = sizeof(T) == 2 && (((int)R.ldo | L.out_col | R.ld_proj | L.off_z) & 3) == 0;
        auto four = [&](int i, const float4& q) {
            if (packed) {
                const float4 w = ((const float4*)nw)[i];
                const float f = inv * L.right_scale;
                float o[4] = {q.x * f * w.x, q.y * f * w.y, q.z * f * w.z, q.w * f * w.w};
                if (gate) {
                    const uint2 g = *(const uint2*)(z + 4 * i);
                    o[0] *= sigmoid_p(__uint_as_float(g.x << 16)); o[1] *= sigmoid_p(__uint_as_float(g.x & 0xffff0000u));
                    o[2] *= sigmoid_p(__uint_as_float(g.y << 16)); o[3] *= sigmoid_p(__uint_as_float(g.y & 0xffff0000u));
                }
                uint2 pk; pk.x = sc_pack(__float2bfloat16(o[0]), __float2bfloat16(o[1])); pk.y = sc_pack(__float2bfloat16(o[2]), __float2bfloat16(o[3]));
                *(uint2*)(out + 4 * i) = pk;
            } else { one(4 * i, q.x, inv); one(4 * i + 1, q.y, inv); one(4 * i + 2, q.z, inv); one(4 * i + 3, q.w, inv); }
        };
#pragma unroll
        for (int j = 0; j < NP_REGS; ++j) if (tid + j * nt < w4) four(tid + j * nt, v[j]);
        for (int i = tid + NP_REGS * nt; i < w4; i += nt) four(i, __ldcg((const float4*)u + i));
        return;
    }
    for (int i = tid; i < w; i += nt) { const float x = __ldcg(u + i); ss += x * x; }
    const float inv = rsqrtf(block_sum(ss, red) / (float)w + L.eps);
    for (int i = tid; i < w; i += nt) one(i, __ldcg(u + i), inv);
}

#define SS_WARPS 8
#define SS_THREADS (SS_WARPS * 32)

// NB: state rows per warp.  U: tokens per turn.  A turn's B and C lie in shared memory, the next one's are on their way to
// registers meanwhile, and the sums over the warps of all its tokens are formed at once, one warp a token: token by token the
// loads, two barriers and the sum came to 0.95 us (200 tokens in fp32, 32 heads of 128 x 64: 190 us a layer).
// The work of CTA (head h, column block by of gy, sequence sq).
template <typename T, int NB, int U>
__device__ __forceinline__ void ssd_step_cta(const MixLayer& L, const MixRun& R, const int h, const int by, const int gy, const int sq) {
    constexpr int NN = SS_WARPS * NB, LD = U * NN / SS_THREADS > 0 ? U * NN / SS_THREADS : 1;      // elements of B (and of C) a thread
    __shared__ float Bs[U * NN], Cs[U * NN], part[U][SS_WARPS][32], red[32];
    __shared__ int s_last;
    if (!R.older) pdl_wait();
    const int p0 = by * 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int grp = h / (L.heads / L.groups), p = p0 + lane;
    const bool pv = p < L.P;
    const int r0 = R.seq_rows[sq], r1 = R.seq_rows[sq + 1];
    const int seq = R.rows[r0].seq;
    float* S = L.state + ((size_t)seq * L.heads + h) * L.N * L.P + p;
    // the state was last written in an earlier step
    float st[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) { const int n = warp + SS_WARPS * i; st[i] = (pv && n < L.N) ? S[(size_t)n * L.P] : 0.f; }
    const float A = rec_rate(L, h), Dh = L.D ? L.D[h] : 0.f, a_const = L.decay ? L.decay[h] : 0.f;
    const bool gated = L.gate == REC_GATE_SILU_NORM;
    pdl_wait();
    if constexpr (U == 1) {
        // one token at a time, as in decode: nothing to overlap, and a turn's detour through registers costs 1 to 5 % (one sequence of
        // 64 heads 8.26 us, by a turn of one 8.48; six 13.9 and 14.5)
        for (int r = r0; r < r1; ++r) {
            const T* xbc = (const T*)R.xbc + (size_t)r * R.ld_xbc;
            for (int n = tid; n < NN; n += SS_THREADS) {
                Bs[n] = n < L.N ? ld_f(xbc + L.rB + grp * L.N + n) : 0.f;
                Cs[n] = n < L.N ? ld_f(xbc + L.rC + grp * L.N + n) : 0.f;
            }
            const float x = pv ? ld_f(xbc + L.rx + h * L.P + p) : 0.f;
            const float dt = rec_dt(L, R, r, h);
            const float z = (gated && warp == 0 && pv) ? ld_f((const T*)R.proj + (size_t)r * R.ld_proj + L.off_z + h * L.P + p) : 0.f;
            const float a = L.decay ? a_const : expf(A * dt), dx = dt * x;
            __syncthreads();
            float y = 0.f;
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const int n = warp + SS_WARPS * i;
                st[i] = fmaf(a, st[i], Bs[n] * dx);
                y = fmaf(st[i], Cs[n], y);
            }
            part[0][warp][lane] = y;
            __syncthreads();
            if (warp == 0 && pv) {
                float s = 0.f;
#pragma unroll
                for (int w = 0; w < SS_WARPS; ++w) s += part[0][w][lane];
                R.ubuf[(size_t)r * R.ld_u + h * L.P + p] = (s + Dh * x) * (gated ? silu_p(z) : 1.f);
            }
        }
    } else {
        float nb[LD], nc[LD], nx[U], ndt[U], nz = 0.f;            // the next turn's
        auto load = [&](int r) {
#pragma unroll
            for (int i = 0; i < LD; ++i) {
                const int e = tid + i * SS_THREADS, u = e / NN, n = e % NN;
                const T* xbc = (const T*)R.xbc + (size_t)(r + u) * R.ld_xbc + grp * L.N + n;
                const bool in = e < U * NN && r + u < r1 && n < L.N;
                nb[i] = in ? ld_f(xbc + L.rB) : 0.f;
                nc[i] = in ? ld_f(xbc + L.rC) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool in = r + u < r1;
                nx[u] = in && pv ? ld_f((const T*)R.xbc + (size_t)(r + u) * R.ld_xbc + L.rx + h * L.P + p) : 0.f;
                ndt[u] = in ? rec_dt(L, R, r + u, h) : 0.f;
            }
            // (the token that this warp sums)
            nz = (gated && warp < U && r + warp < r1 && pv) ? ld_f((const T*)R.proj + (size_t)(r + warp) * R.ld_proj + L.off_z + h * L.P + p) : 0.f;
        };
        auto put = [&]() {
#pragma unroll
            for (int i = 0; i < LD; ++i) {
                const int e = tid + i * SS_THREADS;
                if (e < U * NN) { Bs[e] = nb[i]; Cs[e] = nc[i]; }
            }
        };
        load(r0);
        for (int r = r0; r < r1; r += U) {
            put();
            float x[U], dt[U];
#pragma unroll
            for (int u = 0; u < U; ++u) { x[u] = nx[u]; dt[u] = ndt[u]; }
            const float z = nz;
            __syncthreads();
            if (r + U < r1) load(r + U);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (r + u >= r1) break;
                const float a = L.decay ? a_const : expf(A * dt[u]), dx = dt[u] * x[u];
                float y = 0.f;
#pragma unroll
                for (int i = 0; i < NB; ++i) {
                    const int n = u * NN + warp + SS_WARPS * i;
                    st[i] = fmaf(a, st[i], Bs[n] * dx);
                    y = fmaf(st[i], Cs[n], y);
                }
                part[u][warp][lane] = y;
            }
            __syncthreads();
            if (warp < U && r + warp < r1 && pv) {
                float s = 0.f, xs = x[0];
#pragma unroll
                for (int u = 1; u < U; ++u) if (warp == u) xs = x[u];
#pragma unroll
                for (int w = 0; w < SS_WARPS; ++w) s += part[warp][w][lane];
                R.ubuf[(size_t)(r + warp) * R.ld_u + h * L.P + p] = (s + Dh * xs) * (gated ? silu_p(z) : 1.f);
            }
        }
    }
    if (R.commit) {
#pragma unroll
        for (int i = 0; i < NB; ++i) { const int n = warp + SS_WARPS * i; if (pv && n < L.N) S[(size_t)n * L.P] = st[i]; }
        conv_history_of<T>(L, R, seq, r0, r1, h, p0, 32, tid, SS_THREADS);
    }
    if (!R.fuse_norm) return;
    // ---- the last CTA of a norm part (of the whole row when parts cut through heads) normalises it
    const bool whole = L.heads % L.ngroups != 0;
    const int units = whole ? 1 : L.ngroups, hpu = L.heads / units, unit = h / hpu;
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        int* cnt = R.ssd_counters + sq * units + unit;
        s_last = atomicAdd(cnt, 1) == hpu * gy - 1;
        if (s_last) *cnt = 0;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    for (int r = r0; r < r1; ++r)
        for (int q = 0; q < (whole ? L.ngroups : 1); ++q) norm_part<T>(L, R, r, whole ? q : unit, red);
}

static inline bool ssd_valid(const MixLayer* l) {
    return l->heads >= 1 && l->P >= 1 && l->N >= 1 && l->N <= 256 && l->groups >= 1 && l->heads % l->groups == 0 &&
           l->ngroups >= 1 && (l->heads * l->P) % l->ngroups == 0 && l->taps >= 1 && (l->decay ? l->log_decay != nullptr : l->A_log != nullptr);
}

