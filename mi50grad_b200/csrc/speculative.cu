// Speculative verification on the device: draft chains or trees are checked in ONE
// forward pass and the sequence state afterwards is exactly what feeding only the
// accepted tokens would have produced.
//
// The reference accepts drafts on the host, token by token, and its rollback only
// rewinds a length counter, so rejected drafts stay in the DeltaNet state; its tree
// pass gives every node RoPE position 0 and lets the DeltaNet layers ignore the tree
// (reference: src/inference/speculative.py:231-417, src/inference/tree_speculative.py:296-383,
// src/inference/tp_engine.py:1673-1687,3170-3236).
//
// Four kernels:
//  * deltanet_verify: Gated DeltaNet over a draft tree WITHOUT touching the state.  With S0
//    the committed state, G_t the summed log-decay along node t's path and u_t its rank-1
//    update vector, the state after any path is
//        S_path = exp(G_last) S0 + sum_{a in path} exp(G_last - G_a) k_a u_a^T,
//    so every node needs S0 only through S0^T k_t and S0^T q_t (one pass over the state in
//    registers) plus dot products with its ancestors' keys.  The kernel stages k, u, G and
//    the raw conv inputs of every node for the commit.
//  * spec_accept: greedy acceptance.  Walks the tree from the pending token, following the
//    child whose token equals the model's prediction, advances the sequence length and
//    stores the next pending token.
//  * deltanet_commit: applies the accepted path's rank-1 updates and conv inputs to the
//    state of every linear-attention layer in one launch.
//  * kv_compact: moves the accepted nodes' K/V from slot len+node to slot len+depth in every
//    full-attention layer (a no-op for chains).
#include "kernels.cuh"

#define DN_THREADS 256
#define DN_COLS 32
#define NM SPEC_MAX_NODES

__device__ __forceinline__ int top_bit(unsigned m) { return m ? 31 - __clz(m) : -1; }

#define VF_THREADS 256
#define VF_CHUNK 4               // nodes whose products with the state are reduced together

// One CTA per value head and sequence.  Bound: the states (64 KB a head; 50 MB for 16 sequences of 48 heads), and behind
// them the latencies between the steps, so nothing is done node by node that does not have to be: the convolution, the
// norms, the dot products of all pairs (node, ancestor) and S0^T k, S0^T q of all nodes are formed side by side, and
// only the recursion of the update vectors over a path is serial, per column, without a barrier.  The state stays in
// registers (4 columns x DK / groups rows a thread, read once, 16 bytes at a time) and is requested before anything else.
// Measured for 16 sequences of 5 nodes and 48 heads of 128 x 128: 39 us a layer; a cluster of four CTAs per head
// that walked the nodes with five barriers each took 127.
template <int DK, int DV>
struct VerifySmem {
    static constexpr int NCH = 2 * DK + DV, LPR = DV / 4, RG = VF_THREADS / LPR;
    float cq[NM][DK], ck[NM][DK], cv[NM][DV];             // convolved inputs (unscaled)
    float mm[NM][DV], sq[NM][DV];                         // S0^T k, S0^T q; later the update vectors and the outputs
    float dk[NM][NM], dq[NM][NM];                         // k_t . k_a, q_t . k_a (t == a: k.k, q.k), then their coefficients
    float qq[NM], invq[NM], invk[NM], gl[NM], G[NM], beta[NM], ab[NM][2];
    float eG[NM], eGp[NM], egl[NM];                       // exp of G, of the parent's G, of the node's own log decay
    float ss[NM];
    uchar4 tap[NM];                                       // rows of xraw that hold the inputs at distance 1, 2, 3 on the path
    float abp[VF_THREADS / 32][VF_CHUNK][2];
    unsigned anc[NM];
    alignas(16) __half xraw[NM + 3][NCH];                 // the nodes' inputs; then the history, oldest first
    float4 red[2][VF_CHUNK][RG][LPR];
};

template <int DK, int DV>
__global__ void __launch_bounds__(VF_THREADS, 2) deltanet_verify_kernel(const DeltaParams p, const SpecStage st, int layer) {
    typedef VerifySmem<DK, DV> Smem;
    constexpr int NCH = Smem::NCH, LPR = Smem::LPR, RG = Smem::RG, RPT = DK / RG, WARPS = VF_THREADS / 32;
    constexpr int CB = DV / DN_COLS, HCH = 2 * DK + DN_COLS;          // the history is kept per 32 columns of a head
    extern __shared__ float4 vf_smem[];
    Smem& sm = *(Smem*)vf_smem;
    pdl_launch_dependents();
    if (!p.older) pdl_wait();
    const int j = blockIdx.x, si = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rep = p.nv / p.nk, kh = j / rep;
    const int r0 = p.seq_rows[si], r1 = p.seq_rows[si + 1];
    if (r0 >= r1) return;
    const int N = min(r1 - r0, NM);
    const int seq = p.rows[r0].seq;
    const int rg = tid / LPR, c4 = tid % LPR;                          // rows rg * RPT .., columns 4 c4 ..

    float4 S[RPT];
    const float4* sp = (const float4*)(p.state + (((size_t)seq * p.nv + j) * DK + rg * RPT) * DV) + c4;
    if (((uintptr_t)p.state & 15) == 0) {
#pragma unroll
        for (int i = 0; i < RPT; ++i) S[i] = sp[i * (DV / 4)];
    } else {
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const float* f = (const float*)(sp + i * (DV / 4));
            S[i] = make_float4(f[0], f[1], f[2], f[3]);
        }
    }
    // (histories as well; taps and weights of this thread's channels stay in registers until the convolution)
    auto chan = [&](int c) -> int {
        if (c < DK) return kh * DK + c;
        if (c < 2 * DK) return p.nk * DK + kh * DK + (c - DK);
        return 2 * p.nk * DK + j * DV + (c - 2 * DK);
    };
    constexpr int CPT = (NCH + VF_THREADS - 1) / VF_THREADS;
    __half hist[CPT][3];
    __half cw[CPT][4];
#pragma unroll
    for (int q = 0; q < CPT; ++q) {
        const int c = min(tid + q * VF_THREADS, NCH - 1);
        const int blk = c < 2 * DK ? 0 : (c - 2 * DK) / DN_COLS, hc = c < 2 * DK ? c : 2 * DK + (c - 2 * DK) % DN_COLS;
        const __half* hp = p.conv_state + ((((size_t)seq * p.nv + j) * CB + blk) * HCH + hc) * 3;
#pragma unroll
        for (int e = 0; e < 3; ++e) hist[q][e] = hp[e];
        const __half* w = p.conv_w + (size_t)chan(c) * 4;
#pragma unroll
        for (int e = 0; e < 4; ++e) cw[q][e] = w[e];
    }
    // (and the constants of the last phases, each of which would wait for its own trip there)
    const float a_log = p.A_log[j], dt_bias = __half2float(p.dt_bias[j]), norm_w = __half2float(p.norm_w[tid % DV]);
    static_assert(VF_THREADS % DV == 0, "a thread keeps to one column of the outputs");
#pragma unroll
    for (int q = 0; q < CPT; ++q) {
        const int c = tid + q * VF_THREADS;
        if (c < NCH)
#pragma unroll
            for (int e = 0; e < 3; ++e) sm.xraw[NM + e][c] = hist[q][e];
    }
    pdl_wait();
    constexpr int TZ = VF_THREADS / DV, NZ = 4;                        // gate inputs of the thread's first NZ outputs (nodes TZ apart)
    __half zv[NZ];
#pragma unroll
    for (int q = 0; q < NZ; ++q) zv[q] = p.proj[(size_t)(r0 + min(tid / DV + q * TZ, N - 1)) * p.ld + p.off_z + j * DV + tid % DV];

    auto proj_col = [&](int c) -> int {
        if (c < DK) return p.off_q + kh * DK + c;
        if (c < 2 * DK) return p.off_k + kh * DK + (c - DK);
        return p.off_v + j * DV + (c - 2 * DK);
    };
    if (((p.off_q | p.off_k | p.off_v | p.ld) & 7) == 0 && ((uintptr_t)p.proj & 15) == 0) {
#pragma unroll 2
        for (int i = tid; i < N * (NCH / 8); i += VF_THREADS) {
            const int t = i / (NCH / 8), c = (i - t * (NCH / 8)) * 8;
            *(uint4*)&sm.xraw[t][c] = *(const uint4*)(p.proj + (size_t)(r0 + t) * p.ld + proj_col(c));
        }
    } else {
        for (int i = tid; i < N * NCH; i += VF_THREADS) {
            const int t = i / NCH, c = i - t * NCH;
            sm.xraw[t][c] = p.proj[(size_t)(r0 + t) * p.ld + proj_col(c)];
        }
    }
    // ancestors of a node inside this sequence's block (bit a <-> node a)
    if (tid < N) {
        const unsigned m = (unsigned)(p.rows[r0 + tid].mask & 0xFFFFull) & ((1u << tid) - 1u);
        sm.anc[tid] = m;
        // beyond the root the path goes on in the history
        int row[3];
        unsigned rest = m;
        for (int e = 0, h = NM + 2; e < 3; ++e) {
            const int a = top_bit(rest);
            row[e] = a >= 0 ? a : h--;
            if (a >= 0) rest &= ~(1u << a);
        }
        sm.tap[tid] = make_uchar4((unsigned char)row[0], (unsigned char)row[1], (unsigned char)row[2], 0);
    }
    // ---- a / b inputs of the gates
    const bool inkernel_ab = p.off_a < 0;
    if (inkernel_ab) {
        const __half* wa = p.wa + (size_t)j * p.H;
        const __half* wb = p.wb + (size_t)j * p.H;
        for (int t0 = 0; t0 < N; t0 += VF_CHUNK) {
            float sa[VF_CHUNK], sb[VF_CHUNK];
#pragma unroll
            for (int u = 0; u < VF_CHUNK; ++u) sa[u] = sb[u] = 0.f;
            for (int i = tid * 2; i < p.H; i += VF_THREADS * 2) {
                const float2 av = __half22float2(*(const __half2*)(wa + i)), bv = __half22float2(*(const __half2*)(wb + i));
                float2 ww = make_float2(1.f, 1.f);
                if (p.ln.h) ww = __half22float2(*(const __half2*)(p.ln.w + i));
#pragma unroll
                for (int u = 0; u < VF_CHUNK; ++u) {
                    const int r = r0 + min(t0 + u, N - 1);
                    float2 x = p.ln.h ? *(const float2*)(p.ln.h + (size_t)r * p.ln.H + i) : __half22float2(*(const __half2*)(p.xn + (size_t)r * p.ldx + i));
                    x.x *= ww.x; x.y *= ww.y;
                    sa[u] += x.x * av.x + x.y * av.y;
                    sb[u] += x.x * bv.x + x.y * bv.y;
                }
            }
#pragma unroll
            for (int u = 0; u < VF_CHUNK; ++u) {
                sa[u] = warp_sum(sa[u]);
                sb[u] = warp_sum(sb[u]);
                if (lane == 0) { sm.abp[warp][u][0] = sa[u]; sm.abp[warp][u][1] = sb[u]; }
            }
            __syncthreads();
            if (warp < VF_CHUNK && t0 + warp < N) {
                const int t = t0 + warp;
                const float inv = p.ln.h ? lazy_inv_rms(p.ln, r0 + t, lane) : 1.f;
                float ta = 0.f, tb = 0.f;
#pragma unroll
                for (int w = 0; w < WARPS; ++w) { ta += sm.abp[w][warp][0]; tb += sm.abp[w][warp][1]; }
                if (lane == 0) { sm.ab[t][0] = __half2float(__float2half(ta * inv)); sm.ab[t][1] = __half2float(__float2half(tb * inv)); }
            }
            __syncthreads();
        }
    } else if (tid < N) {
        const __half* pr = p.proj + (size_t)(r0 + tid) * p.ld;
        sm.ab[tid][0] = __half2float(pr[p.off_a + j]);
        sm.ab[tid][1] = __half2float(pr[p.off_b + j]);
    }
    __syncthreads();
    // ---- convolution + SiLU along every node's path: a thread keeps its channel's taps and history
#pragma unroll
    for (int q = 0; q < CPT; ++q) {
        const int c = tid + q * VF_THREADS;
        if (c >= NCH) break;
        const float w0 = __half2float(cw[q][0]), w1 = __half2float(cw[q][1]), w2 = __half2float(cw[q][2]), w3 = __half2float(cw[q][3]);
#pragma unroll 2
        for (int t = 0; t < N; ++t) {
            const uchar4 r = sm.tap[t];
            const float x1 = __half2float(sm.xraw[r.x][c]), x2 = __half2float(sm.xraw[r.y][c]), x3 = __half2float(sm.xraw[r.z][c]);
            const float o = silu_f(x3 * w0 + x2 * w1 + x1 * w2 + __half2float(sm.xraw[t][c]) * w3);
            if (c < DK) sm.cq[t][c] = o; else if (c < 2 * DK) sm.ck[t][c - DK] = o; else sm.cv[t][c - 2 * DK] = o;
        }
    }
    __syncthreads();
    // ---- dot products of every node with itself and with its ancestors, a warp each
    {
        constexpr int E = DK / 32;                        // elements of a lane
        struct alignas(4 * E) Elems { float v[E]; };
        for (int n = warp; n < N * (N + 1) / 2; n += WARPS) {
            int t = (int)((sqrtf(8.f * n + 1.f) - 1.f) * 0.5f);          // pair (t, a), a <= t
            if ((t + 1) * (t + 2) / 2 <= n) ++t;
            if (t * (t + 1) / 2 > n) --t;
            const int a = n - t * (t + 1) / 2;
            if (a != t && !(sm.anc[t] >> a & 1)) continue;
            const Elems ka = *(const Elems*)&sm.ck[a][lane * E], kt = *(const Elems*)&sm.ck[t][lane * E], qt = *(const Elems*)&sm.cq[t][lane * E];
            float kk = 0.f, qk = 0.f, qq = 0.f;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                kk = fmaf(kt.v[e], ka.v[e], kk);
                qk = fmaf(qt.v[e], ka.v[e], qk);
                qq = fmaf(qt.v[e], qt.v[e], qq);
            }
            kk = warp_sum(kk);
            qk = warp_sum(qk);
            if (a == t) qq = warp_sum(qq);
            if (lane == 0) { sm.dk[t][a] = kk; sm.dq[t][a] = qk; if (a == t) sm.qq[t] = qq; }
        }
    }
    __syncthreads();
    if (tid < N) {
        sm.invq[tid] = rsqrtf(sm.qq[tid] + 1e-6f) * rsqrtf((float)DK);
        sm.invk[tid] = rsqrtf(sm.dk[tid][tid] + 1e-6f);
        const float x = sm.ab[tid][0] + dt_bias;
        sm.gl[tid] = fmaxf(-__expf(a_log) * (x > 20.f ? x : log1pf(__expf(x))), -20.f);
        sm.beta[tid] = sigmoid_f(sm.ab[tid][1]);
    }
    __syncthreads();
    if (tid < N) {
        float g = 0.f;                                    // summed log-decay along the path
        for (unsigned m = sm.anc[tid]; m; m &= m - 1) g += sm.gl[__ffs(m) - 1];
        const float own = sm.gl[tid];
        sm.eGp[tid] = __expf(g);                          // (the parent's path is the node's without itself)
        sm.G[tid] = g + own;
        sm.eG[tid] = __expf(g + own);
        sm.egl[tid] = __expf(own);
    }
    // ---- S0^T k and S0^T q of all nodes
    for (int t0 = 0; t0 < N; t0 += VF_CHUNK) {
#pragma unroll 1
        for (int u = 0; u < VF_CHUNK && t0 + u < N; ++u) {
            const float* kp = sm.ck[t0 + u] + rg * RPT;
            const float* qp = sm.cq[t0 + u] + rg * RPT;
            float4 m = make_float4(0.f, 0.f, 0.f, 0.f), q = m;
#pragma unroll
            for (int i = 0; i < RPT; i += 4) {
                const float4 k4 = *(const float4*)(kp + i), q4 = *(const float4*)(qp + i);
                const float kv[4] = {k4.x, k4.y, k4.z, k4.w}, qv[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    m.x = fmaf(S[i + e].x, kv[e], m.x); m.y = fmaf(S[i + e].y, kv[e], m.y); m.z = fmaf(S[i + e].z, kv[e], m.z); m.w = fmaf(S[i + e].w, kv[e], m.w);
                    q.x = fmaf(S[i + e].x, qv[e], q.x); q.y = fmaf(S[i + e].y, qv[e], q.y); q.z = fmaf(S[i + e].z, qv[e], q.z); q.w = fmaf(S[i + e].w, qv[e], q.w);
                }
            }
            sm.red[0][u][rg][c4] = m;
            sm.red[1][u][rg][c4] = q;
        }
        __syncthreads();
        const int cnt = min(VF_CHUNK, N - t0);
        for (int i = tid; i < 2 * cnt * DV; i += VF_THREADS) {
            const int which = i / (cnt * DV), u = (i / DV) % cnt, c = i % DV;
            const float* rp = (const float*)&sm.red[which][u][0][0] + c;
            float s = 0.f;
#pragma unroll
            for (int g = 0; g < RG; ++g) s += rp[g * DV];
            if (which) sm.sq[t0 + u][c] = s * sm.invq[t0 + u]; else sm.mm[t0 + u][c] = s * sm.invk[t0 + u];
        }
        __syncthreads();
    }
    // ---- coefficients of an ancestor's update vector in S_parent^T k_t and in S_t^T q_t
    for (int i = tid; i < N * NM; i += VF_THREADS) {
        const int t = i / NM, a = i % NM;
        const unsigned m = sm.anc[t];
        if (a == t) sm.dq[t][t] *= sm.invq[t] * sm.invk[t];
        else if (m >> a & 1) {
            const float Gp = sm.G[top_bit(m)], Ga = sm.G[a];
            sm.dk[t][a] *= sm.invk[a] * sm.invk[t] * __expf(Gp - Ga);
            sm.dq[t][a] *= sm.invk[a] * sm.invq[t] * __expf(sm.G[t] - Ga);
        }
    }
    __syncthreads();
    // ---- the recursion, one thread per column
    if (tid < DV) {
        for (int t = 0; t < N; ++t) {
            const unsigned m0 = sm.anc[t];
            float Sk = sm.eGp[t] * sm.mm[t][tid], ys = sm.eG[t] * sm.sq[t][tid];
            for (unsigned m = m0; m; m &= m - 1) {
                const int a = __ffs(m) - 1;
                const float u = sm.mm[a][tid];
                Sk = fmaf(sm.dk[t][a], u, Sk);
                ys = fmaf(sm.dq[t][a], u, ys);
            }
            const float delta = (sm.cv[t][tid] - sm.egl[t] * Sk) * sm.beta[t];
            sm.mm[t][tid] = delta;
            sm.sq[t][tid] = fmaf(delta, sm.dq[t][t], ys);
        }
    }
    __syncthreads();
    for (int t = warp; t < N; t += WARPS) {
        float y2 = 0.f;
#pragma unroll
        for (int q = 0; q < DV / 32; ++q) { const float y = sm.sq[t][lane + 32 * q]; y2 = fmaf(y, y, y2); }
        y2 = warp_sum(y2);
        if (lane == 0) sm.ss[t] = rsqrtf(y2 / (float)DV + p.eps);
    }
    __syncthreads();
    // ---- gated RMSNorm over the head's dv outputs; staging for the commit
    unsigned char* blk = st.base + (size_t)layer * st.layer_stride + (size_t)si * st.seq_stride;
    float* su = (float*)(blk + st.off_u);
    {
        const int c = tid % DV;
        int q = 0;
        for (int t = tid / DV; t < N; t += TZ, ++q) {
            __half zh = zv[0];
#pragma unroll
            for (int e = 1; e < NZ; ++e) if (q == e) zh = zv[e];
            if (q >= NZ) zh = p.proj[(size_t)(r0 + t) * p.ld + p.off_z + j * DV + c];
            const float o = sm.sq[t][c] * sm.ss[t] * norm_w * silu_f(__half2float(zh));
            p.out[(size_t)(r0 + t) * p.ldo + j * DV + c] = __float2half(o);
            su[((size_t)t * p.nv + j) * DV + c] = sm.mm[t][c];
        }
    }
    const int conv_dim = 2 * p.nk * DK + p.nv * DV;
    __half* sx = (__half*)(blk + st.off_x);
    const bool key_owner = j % rep == 0;
    for (int i = tid; i < N * NCH; i += VF_THREADS) {
        const int t = i / NCH, c = i - t * NCH;
        if (c >= 2 * DK || key_owner) sx[(size_t)t * conv_dim + chan(c)] = sm.xraw[t][c];
    }
    if (tid < N) ((float*)(blk + st.off_g))[tid * p.nv + j] = sm.G[tid];
    if (key_owner) {
        float* sk = (float*)(blk + st.off_k);
        for (int i = tid; i < N * DK; i += VF_THREADS) {
            const int t = i / DK, e = i - t * DK;
            sk[((size_t)t * p.nk + kh) * DK + e] = sm.ck[t][e] * sm.invk[t];
        }
    }
}

template <int DK, int DV>
static int launch_verify(const DeltaParams* p, const SpecStage* st, int layer, cudaStream_t s) {
    constexpr size_t smem = sizeof(VerifySmem<DK, DV>);
    static SmemOptIn optin;
    if (cudaError_t e = optin.ensure(deltanet_verify_kernel<DK, DV>, smem)) return e;
    return launch_pdl(deltanet_verify_kernel<DK, DV>, dim3(p->nv, p->n_seqs), dim3(VF_THREADS), smem, s, *p, *st, layer);
}

B2_API int b2_deltanet_verify(const DeltaParams* p, const SpecStage* st, int layer, int dk, int dv, cudaStream_t s) {
    if (p->nv % p->nk || !st->base) return cudaErrorInvalidValue;
    if (dk == 128 && dv == 128) return launch_verify<128, 128>(p, st, layer, s);
    if (dk == 64 && dv == 64) return launch_verify<64, 64>(p, st, layer, s);
    return cudaErrorInvalidValue;
}

// Bytes of one staging block and its section offsets.
B2_API long long b2_spec_stage_layout(int nk, int nv, int dk, int dv, int* off_k, int* off_u, int* off_g, int* off_x) {
    auto al = [](long long x) { return (x + 255) & ~255LL; };
    long long o = 0;
    *off_k = (int)o; o = al(o + (long long)NM * nk * dk * 4);
    *off_u = (int)o; o = al(o + (long long)NM * nv * dv * 4);
    *off_g = (int)o; o = al(o + (long long)NM * nv * 4);
    *off_x = (int)o; o = al(o + (long long)NM * (2LL * nk * dk + (long long)nv * dv) * 2);
    return o;
}

// ---------------------------------------------------------------------------
// spec_accept: one thread per sequence (a tree has at most 16 nodes).
// ---------------------------------------------------------------------------
__global__ void spec_accept_kernel(const SpecAcceptParams p) {
    pdl_launch_dependents();
    const int si = blockIdx.x * blockDim.x + threadIdx.x;
    if (si >= p.n_seqs) return;
    int* acc = p.acc + (size_t)si * (NM + 2);
    int* res = p.result + (size_t)si * (NM + 2);
    const int r0 = p.seq_rows[si], r1 = p.seq_rows[si + 1];
    const int N = min(r1 - r0, NM);
    if (N <= 0) { acc[0] = 0; res[0] = -1; return; }
    int parent[NM];
    for (int t = 0; t < N; ++t)
        parent[t] = top_bit((unsigned)(p.rows[r0 + t].mask & 0xFFFFull) & ((1u << t) - 1u));
    int cur = 0, n = 1;
    acc[1] = p.rows[r0].slot;                    // cache slot of the root = length before this step
    acc[2] = 0;
    for (;;) {
        const int pred = p.out_tokens[r0 + cur];
        int nxt = -1;
        for (int t = cur + 1; t < N; ++t)
            if (parent[t] == cur && p.row_tokens[r0 + t] == pred) { nxt = t; break; }
        if (nxt < 0) break;
        res[2 + n - 1] = pred;
        acc[2 + n] = nxt;
        ++n;
        cur = nxt;
    }
    const int next_tok = p.out_tokens[r0 + cur];
    acc[0] = n;
    res[0] = n - 1;
    res[1] = next_tok;
    SeqState* s = p.seqs + p.rows[r0].seq;
    s->len += n;
    s->token = next_tok;
}

B2_API int b2_spec_accept(const SpecAcceptParams* p, cudaStream_t s) {
    if (p->n_seqs < 1) return cudaErrorInvalidValue;
    spec_accept_kernel<<<(p->n_seqs + 31) / 32, 32, 0, s>>>(*p);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// deltanet_commit: grid (dv/32, v heads, layers * sequences)
// ---------------------------------------------------------------------------
template <int DK, int DV>
__global__ void __launch_bounds__(DN_THREADS) deltanet_commit_kernel(const DeltaCommitParams p) {
    constexpr int CB = DV / DN_COLS;
    constexpr int RPT = DK / 8;
    constexpr int NCH = 2 * DK + DN_COLS;
    pdl_launch_dependents();
    const int cb = blockIdx.x, j = blockIdx.y;
    const int layer = blockIdx.z / p.n_seqs, si = blockIdx.z - layer * p.n_seqs;
    const int tid = threadIdx.x, lane = tid & 31, kr = tid >> 5, vcol = lane;
    const int rep = p.nv / p.nk, kh = j / rep;
    const int* acc = p.acc + (size_t)si * (NM + 2);
    const int n = acc[0];
    if (n <= 0) return;
    const int seq = p.rows[p.seq_rows[si]].seq;
    const unsigned char* blk = p.st.base + (size_t)layer * p.st.layer_stride + (size_t)si * p.st.seq_stride;
    const float* sk = (const float*)(blk + p.st.off_k);
    const float* su = (const float*)(blk + p.st.off_u);
    const float* sg = (const float*)(blk + p.st.off_g);
    const __half* sx = (const __half*)(blk + p.st.off_x);

    __shared__ float kp[NM][DK];
    __shared__ float up[NM][DN_COLS];
    __shared__ float coef[NM];
    __shared__ int path[NM];
    if (tid < n) path[tid] = acc[2 + tid];
    __syncthreads();
    const float Gl = sg[path[n - 1] * p.nv + j];
    if (tid < n) coef[tid] = __expf(Gl - sg[path[tid] * p.nv + j]);
    for (int i = tid; i < n * DK; i += DN_THREADS) {
        const int a = i / DK, e = i - a * DK;
        kp[a][e] = sk[((size_t)path[a] * p.nk + kh) * DK + e];
    }
    for (int i = tid; i < n * DN_COLS; i += DN_THREADS) {
        const int a = i / DN_COLS, e = i - a * DN_COLS;
        up[a][e] = su[((size_t)path[a] * p.nv + j) * DV + cb * DN_COLS + e];
    }
    __syncthreads();
    float* sp = p.state0 + (size_t)layer * p.state_layer_stride + (((size_t)seq * p.nv + j) * DK) * DV +
                cb * DN_COLS + vcol;
    float S[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) S[i] = sp[(size_t)(kr + 8 * i) * DV];
    const float g0 = __expf(Gl);
#pragma unroll
    for (int i = 0; i < RPT; ++i) S[i] *= g0;
    for (int a = 0; a < n; ++a) {
        const float cu = coef[a] * up[a][vcol];
#pragma unroll
        for (int i = 0; i < RPT; ++i) S[i] = fmaf(kp[a][kr + 8 * i], cu, S[i]);
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) sp[(size_t)(kr + 8 * i) * DV] = S[i];
    // conv history: the last three inputs of [history, path inputs]
    __half* my_hist = p.conv0 + (size_t)layer * p.conv_layer_stride + ((((size_t)seq * p.nv + j) * CB + cb) * NCH) * 3;
    const int conv_dim = 2 * p.nk * DK + p.nv * DV;
    for (int c = tid; c < NCH; c += DN_THREADS) {
        int ch;
        if (c < DK) ch = kh * DK + c;
        else if (c < 2 * DK) ch = p.nk * DK + kh * DK + (c - DK);
        else ch = 2 * p.nk * DK + j * DV + cb * DN_COLS + (c - 2 * DK);
        __half h[3];
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            const int pos = n + t;               // index into [h0 h1 h2 x_0 .. x_{n-1}], last three
            h[t] = pos < 3 ? my_hist[c * 3 + pos] : sx[(size_t)path[pos - 3] * conv_dim + ch];
        }
#pragma unroll
        for (int t = 0; t < 3; ++t) my_hist[c * 3 + t] = h[t];
    }
}

B2_API int b2_deltanet_commit(const DeltaCommitParams* p, int dk, int dv, cudaStream_t s) {
    if (p->nv % p->nk || p->n_layers < 1 || p->n_seqs < 1) return cudaErrorInvalidValue;
    dim3 grid(dv / DN_COLS, p->nv, p->n_layers * p->n_seqs);
    if (dk == 128 && dv == 128) deltanet_commit_kernel<128, 128><<<grid, DN_THREADS, 0, s>>>(*p);
    else if (dk == 64 && dv == 64) deltanet_commit_kernel<64, 64><<<grid, DN_THREADS, 0, s>>>(*p);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// kv_compact: grid (layers * kv heads, sequences); moves go in increasing depth, each
// destination slot is at or before its source, so earlier moves never clobber later sources.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) kv_compact_kernel(const KvCompactParams p) {
    pdl_launch_dependents();
    const int layer = blockIdx.x / p.nkv, kvh = blockIdx.x - layer * p.nkv, si = blockIdx.y;
    const int* acc = p.acc + (size_t)si * (NM + 2);
    const int n = acc[0];
    if (n <= 1) return;
    const int len0 = acc[1];
    const int seq = p.rows[p.seq_rows[si]].seq;
    const size_t base = (size_t)layer * p.layer_stride + ((size_t)seq * p.max_seq) * p.nkv * p.hd + (size_t)kvh * p.hd;
    const size_t stride = (size_t)p.nkv * p.hd;
    for (int d = 1; d < n; ++d) {
        const int t = acc[2 + d];
        if (t == d) continue;                    // uniform over the CTA
        const size_t src = base + (size_t)(len0 + t) * stride, dst = base + (size_t)(len0 + d) * stride;
        for (int e = threadIdx.x * 2; e < p.hd; e += 256) {
            *(__half2*)(p.k0 + dst + e) = *(const __half2*)(p.k0 + src + e);
            *(__half2*)(p.v0 + dst + e) = *(const __half2*)(p.v0 + src + e);
        }
        __syncthreads();
    }
}

B2_API int b2_kv_compact(const KvCompactParams* p, cudaStream_t s) {
    if (p->n_layers < 1 || p->n_seqs < 1 || (p->hd & 1)) return cudaErrorInvalidValue;
    dim3 grid(p->n_layers * p->nkv, p->n_seqs);
    kv_compact_kernel<<<grid, 128, 0, s>>>(*p);
    return cudaGetLastError();
}
B2_API int b2_sizeof_spec_stage() { return (int)sizeof(SpecStage); }
B2_API int b2_sizeof_spec_accept_params() { return (int)sizeof(SpecAcceptParams); }
B2_API int b2_sizeof_delta_commit_params() { return (int)sizeof(DeltaCommitParams); }
B2_API int b2_sizeof_kv_compact_params() { return (int)sizeof(KvCompactParams); }
