// Gated DeltaNet recurrent step (decode, chain verification, token-serial prefill).
//
// Per value head: causal conv1d(k=4)+SiLU on q,k,v -> L2-normalise q,k ->
// decay = exp(-exp(A_log) softplus(a+dt_bias)), beta = sigmoid(b) ->
//   S <- decay S;  delta = (v - S^T k) beta;  S <- S + k (x) delta;  y = S^T q
// -> y / rms(y) * norm_w * silu(z).  Same math as the reference's fused kernel
// and its CPU oracle (reference: src/kernels/deltanet_v3.hip:70-243,
// src/inference/engine.py:2094-2206); the conv-state shift that the reference
// runs as a second kernel (deltanet_v3.hip:54-65) is folded in.
//
// B200 mapping: the [dk x dv] fp32 state of a head is split by columns over a
// thread-block cluster of dv/32 CTAs (columns evolve independently), which
// gives 4x more CTAs than heads; the only cross-column quantity, sum(y^2) of
// the gated RMSNorm, is exchanged through distributed shared memory.  Each CTA
// keeps a private copy of the conv history of the channels it consumes, so no
// CTA reads history another CTA is shifting.  The state stays in registers
// while a sequence's rows (1 for decode, n for a draft chain or a prompt) are
// consumed in order: one HBM read and one write of the state per launch.
// The tiny a/b projections (2 rows of length hidden per head) can be computed
// in-kernel from the normalised activations, saving a launch.
#include <cooperative_groups.h>
#include <cstdlib>
#include "kernels.cuh"
namespace cg = cooperative_groups;

#define DN_THREADS 256
#define DN_COLS 32


template <int DK, int DV>
__global__ void __launch_bounds__(DN_THREADS) deltanet_step_kernel(const DeltaParams p) {
    constexpr int CB = DV / DN_COLS;
    constexpr int RPT = DK / 8;                  // state rows per thread
    constexpr int NCH = 2 * DK + DN_COLS;        // conv channels this CTA consumes
    cg::cluster_group cluster = cg::this_cluster();
    pdl_launch_dependents();
    if (!p.older) pdl_wait();
    const int cb = blockIdx.x, j = blockIdx.y, si = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, kr = tid >> 5, vcol = lane;
    const int kh = j / (p.nv / p.nk);
    const int r0 = p.seq_rows[si], r1 = p.seq_rows[si + 1];
    if (r0 >= r1) { return; }                    // uniform over the whole cluster
    const int seq = p.rows[r0].seq;

    __shared__ float hist[NCH][3];
    __shared__ float cw[NCH][4];
    __shared__ float cq[DK], ck[DK], cv[DN_COLS];
    __shared__ float red_m[8][DN_COLS], red_q[8][DN_COLS];
    __shared__ float red32[32];
    __shared__ float cl_ss[2];

    // channel id (in the q|k|v conv layout) of local channel c
    auto chan = [&](int c) -> int {
        if (c < DK) return kh * DK + c;
        if (c < 2 * DK) return p.nk * DK + kh * DK + (c - DK);
        return 2 * p.nk * DK + j * DV + cb * DN_COLS + (c - 2 * DK);
    };
    auto proj_col = [&](int c) -> int {
        if (c < DK) return p.off_q + kh * DK + c;
        if (c < 2 * DK) return p.off_k + kh * DK + (c - DK);
        return p.off_v + j * DV + cb * DN_COLS + (c - 2 * DK);
    };
    __half* my_hist = p.conv_state + ((((size_t)seq * p.nv + j) * CB + cb) * NCH) * 3;
    for (int c = tid; c < NCH; c += DN_THREADS) {
#pragma unroll
        for (int t = 0; t < 3; ++t) hist[c][t] = __half2float(my_hist[c * 3 + t]);
        const __half* w = p.conv_w + (size_t)chan(c) * 4;
#pragma unroll
        for (int t = 0; t < 4; ++t) cw[c][t] = __half2float(w[t]);
    }
    float S[RPT];
    float* sp = p.state + (((size_t)seq * p.nv + j) * DK) * DV + cb * DN_COLS + vcol;
#pragma unroll
    for (int i = 0; i < RPT; ++i) S[i] = sp[(size_t)(kr + 8 * i) * DV];
    const float neg_expA = -__expf(p.A_log[j]);
    const float dtb = __half2float(p.dt_bias[j]);
    const float nw = __half2float(p.norm_w[cb * DN_COLS + vcol]);
    // The a/b projections' weights (times the norm weights of a lazily normalised input) do not depend on
    // this step either: the first DN_PRE pairs per thread wait in registers.
    constexpr int DN_PRE = 10;
    const bool inkernel_ab = p.off_a < 0;
    float2 pa[DN_PRE], pb[DN_PRE];
#pragma unroll
    for (int k = 0; k < DN_PRE; ++k) {
        pa[k] = pb[k] = make_float2(0.f, 0.f);
        const int i = tid * 2 + k * DN_THREADS * 2;
        if (inkernel_ab && i < p.H) {
            float2 av = __half22float2(*(const __half2*)(p.wa + (size_t)j * p.H + i));
            float2 bv = __half22float2(*(const __half2*)(p.wb + (size_t)j * p.H + i));
            if (p.ln.h) {
                const float2 ww = __half22float2(*(const __half2*)(p.ln.w + i));
                av.x *= ww.x; av.y *= ww.y; bv.x *= ww.x; bv.y *= ww.y;
            }
            pa[k] = av; pb[k] = bv;
        }
    }
    __syncthreads();
    // Everything above (conv history, state slice, weights) was left by earlier steps; what follows reads
    // this step's in-projection output and residual stream.
    pdl_wait();

    for (int r = r0; r < r1; ++r) {
        const __half* pr = p.proj + (size_t)r * p.ld;
        // ---- phase A (no barrier inside): conv + SiLU of this CTA's channels, partial sums of the
        // a/b projections.  With a lazily normalised input the 1/rms factor is applied to the
        // finished dot products, so nothing here waits on it.
        float sa = 0.f, sb = 0.f;
        if (inkernel_ab) {
            const __half* wa = p.wa + (size_t)j * p.H;
            const __half* wb = p.wb + (size_t)j * p.H;
            if (p.ln.h) {
                const float* hr = p.ln.h + (size_t)r * p.ln.H;
                float2 hv[DN_PRE];
#pragma unroll
                for (int k = 0; k < DN_PRE; ++k) {
                    const int i = tid * 2 + k * DN_THREADS * 2;
                    hv[k] = i < p.H ? *(const float2*)(hr + i) : make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int k = 0; k < DN_PRE; ++k) {
                    sa += hv[k].x * pa[k].x + hv[k].y * pa[k].y;
                    sb += hv[k].x * pb[k].x + hv[k].y * pb[k].y;
                }
                for (int i = tid * 2 + DN_PRE * DN_THREADS * 2; i < p.H; i += DN_THREADS * 2) {
                    float2 hv2 = *(const float2*)(hr + i);
                    float2 ww = __half22float2(*(const __half2*)(p.ln.w + i));
                    float2 av = __half22float2(*(const __half2*)(wa + i));
                    float2 bv = __half22float2(*(const __half2*)(wb + i));
                    float x0 = hv2.x * ww.x, x1 = hv2.y * ww.y;
                    sa += x0 * av.x + x1 * av.y;
                    sb += x0 * bv.x + x1 * bv.y;
                }
            } else {
                const __half* x = p.xn + (size_t)r * p.ldx;
                float2 xv[DN_PRE];
#pragma unroll
                for (int k = 0; k < DN_PRE; ++k) {
                    const int i = tid * 2 + k * DN_THREADS * 2;
                    xv[k] = i < p.H ? __half22float2(*(const __half2*)(x + i)) : make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int k = 0; k < DN_PRE; ++k) {
                    sa += xv[k].x * pa[k].x + xv[k].y * pa[k].y;
                    sb += xv[k].x * pb[k].x + xv[k].y * pb[k].y;
                }
                for (int i = tid * 2 + DN_PRE * DN_THREADS * 2; i < p.H; i += DN_THREADS * 2) {
                    float2 xv2 = __half22float2(*(const __half2*)(x + i));
                    float2 av = __half22float2(*(const __half2*)(wa + i));
                    float2 bv = __half22float2(*(const __half2*)(wb + i));
                    sa += xv2.x * av.x + xv2.y * av.y;
                    sb += xv2.x * bv.x + xv2.y * bv.y;
                }
            }
            sa = warp_sum(sa);
            sb = warp_sum(sb);
            if (lane == 0) { red_m[kr][0] = sa; red_m[kr][1] = sb; }
        }
        for (int c = tid; c < NCH; c += DN_THREADS) {
            float x = __half2float(pr[proj_col(c)]);
            float o = hist[c][0] * cw[c][0] + hist[c][1] * cw[c][1] + hist[c][2] * cw[c][2] + x * cw[c][3];
            hist[c][0] = hist[c][1]; hist[c][1] = hist[c][2]; hist[c][2] = x;
            o = silu_f(o);
            if (c < DK) cq[c] = o; else if (c < 2 * DK) ck[c - DK] = o; else cv[c - 2 * DK] = o;
        }
        __syncthreads();
        // ---- phase B: warps 0..2 the q/k norms and q.k, warp 3 the a/b inputs
        if (kr < 3) {
            float s = 0.f;
            for (int i = lane; i < DK; i += 32) {
                float a = (kr == 1) ? ck[i] : cq[i], b = (kr == 0) ? cq[i] : ck[i];
                s += a * b;                      // kr0: q.q  kr1: k.k  kr2: q.k
            }
            s = warp_sum(s);
            if (lane == 0) red32[kr] = s;
        } else if (kr == 3) {
            float a_in, b_in;
            if (inkernel_ab) {
                float inv = p.ln.h ? lazy_inv_rms(p.ln, r, lane) : 1.f;
                float ta = 0.f, tb = 0.f;
#pragma unroll
                for (int w = 0; w < 8; ++w) { ta += red_m[w][0]; tb += red_m[w][1]; }
                // the unfused path rounds the projection output to fp16: keep that rounding
                a_in = __half2float(__float2half(ta * inv));
                b_in = __half2float(__float2half(tb * inv));
            } else {
                a_in = __half2float(pr[p.off_a + j]);
                b_in = __half2float(pr[p.off_b + j]);
            }
            if (lane == 0) { red32[3] = a_in; red32[4] = b_in; }
        }
        __syncthreads();
        const float invq = rsqrtf(red32[0] + 1e-6f) * rsqrtf((float)DK);
        const float invk = rsqrtf(red32[1] + 1e-6f);
        const float kq = red32[2] * invq * invk;
        const float a_in = red32[3], b_in = red32[4];
        float gl = neg_expA * (a_in + dtb > 20.f ? a_in + dtb : log1pf(__expf(a_in + dtb)));
        gl = fmaxf(gl, -20.f);
        const float decay = __expf(gl);
        const float beta = sigmoid_f(b_in);
        // ---- phase C: single pass over the state slice: m = S^T k, sq = S^T q
        float mp = 0.f, qp = 0.f;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            mp = fmaf(S[i], ck[kr + 8 * i], mp);
            qp = fmaf(S[i], cq[kr + 8 * i], qp);
        }
        red_m[kr][vcol] = mp * invk;
        red_q[kr][vcol] = qp * invq;
        __syncthreads();
        float mm = 0.f, sq = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) { mm += red_m[w][vcol]; sq += red_q[w][vcol]; }
        const float delta = (cv[vcol] - decay * mm) * beta;
        const float y = decay * sq + delta * kq;
#pragma unroll
        for (int i = 0; i < RPT; ++i) S[i] = decay * S[i] + ck[kr + 8 * i] * invk * delta;
        // ---- gated RMSNorm over the head's dv outputs (dv/32 CTAs of the cluster)
        float ss = warp_sum(y * y);              // every warp holds the same y per column
        const int slot = (r - r0) & 1;
        if (tid == 0) cl_ss[slot] = ss;
        cluster.sync();
        float tot = 0.f;
#pragma unroll
        for (int c = 0; c < CB; ++c) tot += *cluster.map_shared_rank(&cl_ss[slot], c);
        if (kr == 0) {
            float z = __half2float(pr[p.off_z + j * DV + cb * DN_COLS + vcol]);
            float o = y * rsqrtf(tot / (float)DV + p.eps) * nw * silu_f(z);
            p.out[(size_t)r * p.ldo + j * DV + cb * DN_COLS + vcol] = __float2half(o);
        }
        // the cluster barrier above also orders this row's shared-memory reads before the next row's writes
    }
    cluster.sync();                              // no CTA leaves while a peer may still read its shared memory
    if (!p.commit) return;
#pragma unroll
    for (int i = 0; i < RPT; ++i) sp[(size_t)(kr + 8 * i) * DV] = S[i];
    for (int c = tid; c < NCH; c += DN_THREADS)
#pragma unroll
        for (int t = 0; t < 3; ++t) my_hist[c * 3 + t] = __float2half(hist[c][t]);
}

// ---------------------------------------------------------------------------
// One CTA per value head (all DV columns: DV/32 groups of four warps).  Same arithmetic and the same
// state / conv-history layout as deltanet_step_kernel, laid out for latency: a decode step is a chain of
// short dependent phases, so (1) the sum over the head's columns for the gated RMSNorm goes through shared
// memory instead of a cluster barrier, (2) everything that earlier steps left (state slice, conv history,
// weights of the a/b projections) is in registers before the dependency wait, and (3) all loads that
// depend on this step's in-projection are issued together right after it.
// ---------------------------------------------------------------------------
template <int DK, int DV>
__global__ void __launch_bounds__(DV / 32 * 128) deltanet_head_kernel(const DeltaParams p) {
    constexpr int CB = DV / DN_COLS;
    constexpr int KR = 4;                        // warps sharing one 32-column block: state rows kr, kr + KR, ...
    constexpr int NT = CB * KR * 32;
    constexpr int RPT = DK / KR;                 // state rows per thread
    constexpr int NCHB = 2 * DK + DN_COLS;       // channels per private history copy in memory
    constexpr int NCH = 2 * DK + DV;             // conv channels of the head: q | k | v
    constexpr int PRE = 5;                       // a/b weight pairs per thread kept in registers
    pdl_launch_dependents();
    if (!p.older) pdl_wait();
    const int j = blockIdx.x, si = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cb = warp / KR, kr = warp % KR, col = cb * DN_COLS + lane;
    const int kh = j / (p.nv / p.nk);
    const int r0 = p.seq_rows[si], r1 = p.seq_rows[si + 1];
    if (r0 >= r1) return;
    const int seq = p.rows[r0].seq;

    __shared__ float cq[DK], ck[DK], cv[DV];
    __shared__ float red_m[KR][DV], red_q[KR][DV];
    __shared__ float red_ab[NT / 32][2];
    __shared__ float red32[8];
    __shared__ float ss_cb[CB];

    // ---- left by earlier steps: conv history + weights of this thread's channel, state slice, constants
    const bool has_ch = tid < NCH;
    int pcol = 0;
    float h0 = 0.f, h1 = 0.f, h2 = 0.f, w0 = 0.f, w1 = 0.f, w2 = 0.f, w3 = 0.f;
    __half* hist_base = p.conv_state + (((size_t)seq * p.nv + j) * CB) * NCHB * 3;
    __half* my_hist = nullptr;
    if (has_ch) {
        int gch;
        if (tid < DK) { gch = kh * DK + tid; pcol = p.off_q + kh * DK + tid; my_hist = hist_base + (size_t)tid * 3; }
        else if (tid < 2 * DK) { gch = p.nk * DK + kh * DK + (tid - DK); pcol = p.off_k + kh * DK + (tid - DK); my_hist = hist_base + (size_t)tid * 3; }
        else {
            const int v = tid - 2 * DK;
            gch = 2 * p.nk * DK + j * DV + v; pcol = p.off_v + j * DV + v;
            my_hist = hist_base + ((size_t)(v / DN_COLS) * NCHB + 2 * DK + (v % DN_COLS)) * 3;
        }
        h0 = __half2float(my_hist[0]); h1 = __half2float(my_hist[1]); h2 = __half2float(my_hist[2]);
        const __half* w = p.conv_w + (size_t)gch * 4;
        w0 = __half2float(w[0]); w1 = __half2float(w[1]); w2 = __half2float(w[2]); w3 = __half2float(w[3]);
    }
    float S[RPT];
    float* sp = p.state + (((size_t)seq * p.nv + j) * DK) * DV + col;
#pragma unroll
    for (int i = 0; i < RPT; ++i) S[i] = sp[(size_t)(kr + KR * i) * DV];
    const float neg_expA = -__expf(p.A_log[j]);
    const float dtb = __half2float(p.dt_bias[j]);
    const float nw = __half2float(p.norm_w[col]);
    const bool inkernel_ab = p.off_a < 0;
    float2 pa[PRE], pb[PRE];
#pragma unroll
    for (int k = 0; k < PRE; ++k) {
        pa[k] = pb[k] = make_float2(0.f, 0.f);
        const int i = tid * 2 + k * NT * 2;
        if (inkernel_ab && i < p.H) {
            float2 av = __half22float2(*(const __half2*)(p.wa + (size_t)j * p.H + i));
            float2 bv = __half22float2(*(const __half2*)(p.wb + (size_t)j * p.H + i));
            if (p.ln.h) {
                const float2 ww = __half22float2(*(const __half2*)(p.ln.w + i));
                av.x *= ww.x; av.y *= ww.y; bv.x *= ww.x; bv.y *= ww.y;
            }
            pa[k] = av; pb[k] = bv;
        }
    }
    pdl_wait();

    for (int r = r0; r < r1; ++r) {
        const __half* pr = p.proj + (size_t)r * p.ld;
        // ---- every load that depends on this step, issued together
        float2 xin[PRE];
#pragma unroll
        for (int k = 0; k < PRE; ++k) {
            xin[k] = make_float2(0.f, 0.f);
            const int i = tid * 2 + k * NT * 2;
            if (inkernel_ab && i < p.H)
                xin[k] = p.ln.h ? *(const float2*)(p.ln.h + (size_t)r * p.ln.H + i)
                                : __half22float2(*(const __half2*)(p.xn + (size_t)r * p.ldx + i));
        }
        const float xc = has_ch ? __half2float(pr[pcol]) : 0.f;
        const float z = kr == 0 ? __half2float(pr[p.off_z + j * DV + col]) : 0.f;
        float ssp = 0.f, a_dir = 0.f, b_dir = 0.f;
        if (warp == 3) {
            if (inkernel_ab && p.ln.h) for (int i = lane; i < p.ln.np; i += 32) ssp += p.ln.ss[(size_t)r * p.ln.np + i];
            if (!inkernel_ab) { a_dir = __half2float(pr[p.off_a + j]); b_dir = __half2float(pr[p.off_b + j]); }
        }
        // ---- phase A: partial sums of the a/b projections, conv + SiLU of this thread's channel
        if (inkernel_ab) {
            float sa = 0.f, sb = 0.f;
#pragma unroll
            for (int k = 0; k < PRE; ++k) {
                sa += xin[k].x * pa[k].x + xin[k].y * pa[k].y;
                sb += xin[k].x * pb[k].x + xin[k].y * pb[k].y;
            }
            for (int i = tid * 2 + PRE * NT * 2; i < p.H; i += NT * 2) {        // hidden sizes beyond PRE pairs per thread
                float2 xv = p.ln.h ? *(const float2*)(p.ln.h + (size_t)r * p.ln.H + i)
                                   : __half22float2(*(const __half2*)(p.xn + (size_t)r * p.ldx + i));
                float2 av = __half22float2(*(const __half2*)(p.wa + (size_t)j * p.H + i));
                float2 bv = __half22float2(*(const __half2*)(p.wb + (size_t)j * p.H + i));
                if (p.ln.h) {
                    const float2 ww = __half22float2(*(const __half2*)(p.ln.w + i));
                    av.x *= ww.x; av.y *= ww.y; bv.x *= ww.x; bv.y *= ww.y;
                }
                sa += xv.x * av.x + xv.y * av.y;
                sb += xv.x * bv.x + xv.y * bv.y;
            }
            sa = warp_sum(sa);
            sb = warp_sum(sb);
            if (lane == 0) { red_ab[warp][0] = sa; red_ab[warp][1] = sb; }
        }
        if (has_ch) {
            float o = silu_f(h0 * w0 + h1 * w1 + h2 * w2 + xc * w3);
            h0 = h1; h1 = h2; h2 = xc;
            if (tid < DK) cq[tid] = o; else if (tid < 2 * DK) ck[tid - DK] = o; else cv[tid - 2 * DK] = o;
        }
        __syncthreads();
        // ---- phase B: warps 0..2 the q/k norms and q.k, warp 3 the a/b inputs
        if (warp < 3) {
            float s = 0.f;
            for (int i = lane; i < DK; i += 32) {
                float a = (warp == 1) ? ck[i] : cq[i], b = (warp == 0) ? cq[i] : ck[i];
                s += a * b;                      // warp 0: q.q  warp 1: k.k  warp 2: q.k
            }
            s = warp_sum(s);
            if (lane == 0) red32[warp] = s;
        } else if (warp == 3) {
            float a_in = a_dir, b_in = b_dir;
            if (inkernel_ab) {
                float inv = 1.f;
                if (p.ln.h) inv = rsqrtf(warp_sum(ssp) / (float)p.ln.H + p.ln.eps);
                float ta = 0.f, tb = 0.f;
                for (int w = lane; w < NT / 32; w += 32) { ta += red_ab[w][0]; tb += red_ab[w][1]; }
                ta = warp_sum(ta); tb = warp_sum(tb);
                // the unfused path rounds the projection output to fp16: keep that rounding
                a_in = __half2float(__float2half(ta * inv));
                b_in = __half2float(__float2half(tb * inv));
            }
            if (lane == 0) { red32[3] = a_in; red32[4] = b_in; }
        }
        __syncthreads();
        const float invq = rsqrtf(red32[0] + 1e-6f) * rsqrtf((float)DK);
        const float invk = rsqrtf(red32[1] + 1e-6f);
        const float kq = red32[2] * invq * invk;
        const float a_in = red32[3], b_in = red32[4];
        float gl = neg_expA * (a_in + dtb > 20.f ? a_in + dtb : log1pf(__expf(a_in + dtb)));
        gl = fmaxf(gl, -20.f);
        const float decay = __expf(gl);
        const float beta = sigmoid_f(b_in);
        // ---- phase C: single pass over the state slice: m = S^T k, sq = S^T q
        float mp = 0.f, qp = 0.f;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            mp = fmaf(S[i], ck[kr + KR * i], mp);
            qp = fmaf(S[i], cq[kr + KR * i], qp);
        }
        red_m[kr][col] = mp * invk;
        red_q[kr][col] = qp * invq;
        __syncthreads();
        float mm = 0.f, sq = 0.f;
#pragma unroll
        for (int w = 0; w < KR; ++w) { mm += red_m[w][col]; sq += red_q[w][col]; }
        const float delta = (cv[col] - decay * mm) * beta;
        const float y = decay * sq + delta * kq;
#pragma unroll
        for (int i = 0; i < RPT; ++i) S[i] = decay * S[i] + ck[kr + KR * i] * invk * delta;
        // ---- gated RMSNorm over the head's DV outputs
        const float ss = warp_sum(y * y);
        if (kr == 0 && lane == 0) ss_cb[cb] = ss;
        __syncthreads();
        if (kr == 0) {
            float tot = 0.f;
#pragma unroll
            for (int c = 0; c < CB; ++c) tot += ss_cb[c];
            float o = y * rsqrtf(tot / (float)DV + p.eps) * nw * silu_f(z);
            p.out[(size_t)r * p.ldo + j * DV + col] = __float2half(o);
        }
        __syncthreads();                         // this row's shared-memory reads before the next row's writes
    }
    if (!p.commit) return;
#pragma unroll
    for (int i = 0; i < RPT; ++i) sp[(size_t)(kr + KR * i) * DV] = S[i];
    if (has_ch) {
        const __half a0 = __float2half(h0), a1 = __float2half(h1), a2 = __float2half(h2);
        if (tid < 2 * DK) {
            // q / k history: every column block keeps its own copy (the chunked scan and the verify kernels read them)
#pragma unroll
            for (int c = 0; c < CB; ++c) {
                __half* d = hist_base + ((size_t)c * NCHB + tid) * 3;
                d[0] = a0; d[1] = a1; d[2] = a2;
            }
        } else {
            my_hist[0] = a0; my_hist[1] = a1; my_hist[2] = a2;
        }
    }
}

template <int DK, int DV>
static int launch_delta_head(const DeltaParams* p, cudaStream_t s) {
    return launch_pdl(deltanet_head_kernel<DK, DV>, dim3(p->nv, p->n_seqs), dim3(DV / 32 * 128), 0, s, *p);
}

template <int DK, int DV>
static int launch_delta(const DeltaParams* p, cudaStream_t s) {
    constexpr int CB = DV / DN_COLS;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CB, p->nv, p->n_seqs);
    cfg.blockDim = dim3(DN_THREADS);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CB;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    // programmatic dependent launch: the CTAs become resident, load their state slice, conv history and
    // weights while the in-projection is still finishing, and wait (griddepcontrol.wait) only then
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, deltanet_step_kernel<DK, DV>, *p);
}

B2_API int b2_deltanet_step(const DeltaParams* p, int dk, int dv, cudaStream_t s) {
    if (p->nv % p->nk) return cudaErrorInvalidValue;
    // one CTA per head (deltanet_head_kernel) unless B200GRAD_DELTANET_CLUSTER selects the cluster form
    static const bool cluster_form = getenv("B200GRAD_DELTANET_CLUSTER") != nullptr;
    if (!cluster_form) {
        if (dk == 128 && dv == 128) return launch_delta_head<128, 128>(p, s);
        if (dk == 64 && dv == 64) return launch_delta_head<64, 64>(p, s);
    }
    if (dk == 128 && dv == 128) return launch_delta<128, 128>(p, s);
    if (dk == 64 && dv == 64) return launch_delta<64, 64>(p, s);
    return cudaErrorInvalidValue;
}
B2_API int b2_sizeof_delta_params() { return (int)sizeof(DeltaParams); }
B2_API int b2_delta_conv_channels(int dk) { return 2 * dk + DN_COLS; }

// ===========================================================================
// Chunked Gated DeltaNet scan (prefill, long draft chains).
//
// The reference has no chunked form: its prefill loops the decode kernel token by token
// (reference: src/inference/engine.py:3141-3161).  Here a sequence is consumed in chunks of
// 64 rows.  With G_i the running sum of the log-decays inside a chunk and S0 the state at its
// start:
//     A[i][j] = beta_i exp(G_i-G_j) (k_i.k_j)  (j <  i)      W[i][j] = exp(G_i-G_j) (q_i.k_j)  (j <= i)
//     (I + A) U = beta (V - exp(G) K S0)                     (forward substitution, blocked by 8 rows)
//     Y  = exp(G) Q S0 + W U
//     S' = exp(G_C) S0 + (exp(G_C-G) K)^T U
// Same decomposition as the step kernel: a cluster of dv/32 CTAs per value head, each owning
// 32 state columns (columns never interact except through sum(y^2) of the gated RMSNorm,
// which is exchanged through distributed shared memory once per chunk).  All matrices of a
// chunk live in shared memory in fp32; the state slice stays in registers across chunks.
// ===========================================================================
#define DC_C 32                  // rows per chunk: small enough that two CTAs share an SM and overlap their phases
#define DC_LDK(DK) ((DK) + 4)    // padded row stride of the q/k tiles (conflict-free fragment loads)
#define DC_LDA (DC_C + 4)
#define DC_LDU (DN_COLS + 8)     // row stride of U and of the state copy (they are B operands)

// The matrix products of a chunk run on the tensor cores as TF32 (fp32 storage, 10-bit
// mantissa: the precision of the fp16 activations the inputs come from), accumulating in fp32.
__device__ __forceinline__ float tf32r(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], float a0, float a1, float a2, float a3, float b0, float b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(__float_as_uint(a0)), "r"(__float_as_uint(a1)), "r"(__float_as_uint(a2)), "r"(__float_as_uint(a3)),
                   "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}

// Four 8x4 fp32 tiles in one instruction: lane l supplies the address of row (l & 7) of tile l >> 3
// (16 bytes = 4 floats per row); afterwards every lane holds element (lane >> 2, lane & 3) of each
// tile, which is exactly the TF32 fragment layout of mma.m16n8k8.
__device__ __forceinline__ void ldsm4(float (&r)[4], const float* row_ptr) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(row_ptr);
    uint32_t x0, x1, x2, x3;
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(x0), "=r"(x1), "=r"(x2), "=r"(x3) : "r"(a));
    r[0] = __uint_as_float(x0); r[1] = __uint_as_float(x1); r[2] = __uint_as_float(x2); r[3] = __uint_as_float(x3);
}
__device__ __forceinline__ void ldsm2(float (&r)[2], const float* row_ptr) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(row_ptr);
    uint32_t x0, x1;
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(x0), "=r"(x1) : "r"(a));
    r[0] = __uint_as_float(x0); r[1] = __uint_as_float(x1);
}
__device__ __forceinline__ float silu_fast(float x) { return __fdividef(x, 1.f + __expf(-x)); }

template <int DK, int DV>
__global__ void __launch_bounds__(DN_THREADS, 2) deltanet_chunk_kernel(const DeltaParams p, const __half* __restrict__ ab, int ld_ab,
                                                                      const __half* __restrict__ qk_pre, int ld_qk) {
    constexpr int CB = DV / DN_COLS;
    constexpr int MT = DK / 16;               // 16-row tiles of the state slice, one or two per warp
    constexpr int SPW = (MT + 7) / 8;         // state m-tiles per warp
    constexpr int NCH = 2 * DK + DN_COLS;
    constexpr int LDK = DC_LDK(DK);
    static_assert(DK % 16 == 0 && MT <= 16, "state tiling");
    cg::cluster_group cluster = cg::this_cluster();
    pdl_launch_dependents();
    const int cb = blockIdx.x, j = blockIdx.y, si = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, kr = tid >> 5, vcol = lane;
    const int g = lane >> 2, t = lane & 3;    // fragment coordinates
    const int kh = j / (p.nv / p.nk);
    const int r0 = p.seq_rows[si], r1 = p.seq_rows[si + 1];
    if (r0 >= r1) return;
    const int seq = p.rows[r0].seq;

    extern __shared__ __align__(16) float dsm[];
    float* Qs = dsm;                          // [C][LDK]
    float* Ks = Qs + DC_C * LDK;              // [C][LDK]
    float* Us = Ks + DC_C * LDK;              // [C][LDU]  v -> b -> u (in place)
    float* QSs = Us + DC_C * DC_LDU;          // [C][32]   exp(G) Q S0
    float* Ys = QSs + DC_C * DN_COLS;         // [C][32]
    float* As = Ys + DC_C * DN_COLS;          // [C][LDA]
    float* Ws = As + DC_C * DC_LDA;           // [C][LDA]
    float* S0t = Ws + DC_C * DC_LDA;          // [32][LDK]  transposed copy of the state slice (a B operand)
    float* hist = S0t + DN_COLS * LDK;        // [NCH][3]
    float* cw = hist + NCH * 3;               // [NCH][4]
    float* Gs = cw + NCH * 4;                 // [C] running log-decay
    float* bs = Gs + DC_C;                    // [C] beta
    float* gs = bs + DC_C;                    // [C] log-decay per row
    float* cl_ss = gs + DC_C;                 // [2][C]
    __half* Xr = (__half*)(cl_ss + 2 * DC_C);  // [C+3][NCH] raw conv inputs of the chunk (3 history rows first)

    auto chan = [&](int c) -> int {
        if (c < DK) return kh * DK + c;
        if (c < 2 * DK) return p.nk * DK + kh * DK + (c - DK);
        return 2 * p.nk * DK + j * DV + cb * DN_COLS + (c - 2 * DK);
    };
    auto proj_col = [&](int c) -> int {
        if (c < DK) return p.off_q + kh * DK + c;
        if (c < 2 * DK) return p.off_k + kh * DK + (c - DK);
        return p.off_v + j * DV + cb * DN_COLS + (c - 2 * DK);
    };
    __half* my_hist = p.conv_state + ((((size_t)seq * p.nv + j) * CB + cb) * NCH) * 3;
    for (int c = tid; c < NCH; c += DN_THREADS) {
#pragma unroll
        for (int q = 0; q < 3; ++q) hist[c * 3 + q] = __half2float(my_hist[c * 3 + q]);
        const __half* w = p.conv_w + (size_t)chan(c) * 4;
#pragma unroll
        for (int q = 0; q < 4; ++q) cw[c * 4 + q] = __half2float(w[q]);
    }
    // The state slice [DK x 32] lives in registers as accumulator fragments: warp w owns the
    // 16-row tiles w (and w + 8), each as four 16x8 tiles: S[m][n][0..3] = rows g / g+8, cols 2t / 2t+1.
    float S[SPW][4][4];
    float* sp = p.state + (((size_t)seq * p.nv + j) * DK) * DV + cb * DN_COLS;
#pragma unroll
    for (int m = 0; m < SPW; ++m) {
        const int mt = kr + 8 * m;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            if (mt < MT) {
                const float2 lo = *(const float2*)(sp + (size_t)(16 * mt + g) * DV + 8 * n + 2 * t);
                const float2 hi = *(const float2*)(sp + (size_t)(16 * mt + g + 8) * DV + 8 * n + 2 * t);
                S[m][n][0] = lo.x; S[m][n][1] = lo.y; S[m][n][2] = hi.x; S[m][n][3] = hi.y;
            } else {
                S[m][n][0] = S[m][n][1] = S[m][n][2] = S[m][n][3] = 0.f;
            }
        }
    }
    const float neg_expA = -__expf(p.A_log[j]);
    const float dtb = __half2float(p.dt_bias[j]);
    const float nw = __half2float(p.norm_w[cb * DN_COLS + vcol]);
    const float qscale = rsqrtf((float)DK);
    __syncthreads();

    // raw-tile staging: 16-byte cp.async pieces; rows before the sequence start come from the saved history,
    // rows past its end are zero
    auto stage_raw = [&](int rb_) {
        constexpr int PPR = NCH / 8;                       // 16-byte pieces per row
        for (int idx = tid; idx < (DC_C + 3) * PPR; idx += DN_THREADS) {
            const int row = idx / PPR, pc = idx % PPR;
            const int c = pc * 8;
            const int ri = rb_ - 3 + row;
            __half* dst = Xr + row * NCH + c;
            if (qk_pre && c < 2 * DK) {
                // q / k columns: convolved, normalised (q also scaled) rows from the pre-pass; no history rows
                if (ri >= rb_ && ri < r1)
                    cp_async16(dst, qk_pre + (size_t)(ri - r0) * ld_qk + (c < DK ? kh * DK + c : p.nk * DK + kh * DK + (c - DK)));
                else
                    *(uint4*)dst = make_uint4(0u, 0u, 0u, 0u);
            } else if (ri >= r0 && ri < r1) {
                cp_async16(dst, p.proj + (size_t)ri * p.ld + proj_col(c));
            } else if (ri < r0) {
#pragma unroll
                for (int e = 0; e < 8; ++e) dst[e] = __float2half(hist[(c + e) * 3 + (ri - r0 + 3)]);
            } else {
                *(uint4*)dst = make_uint4(0u, 0u, 0u, 0u);
            }
        }
        cp_async_commit();
    };
    stage_raw(r0);
    // the gate inputs of a chunk are fetched one chunk ahead (a global round trip off the critical path)
    float a_pre = 0.f, b_pre = 0.f;
    auto fetch_gates = [&](int rb_) {
        a_pre = b_pre = 0.f;
        if (tid < DC_C && rb_ + tid < r1) {
            const __half* abr = ab + (size_t)(rb_ + tid) * ld_ab;
            a_pre = __half2float(abr[j]); b_pre = __half2float(abr[p.nv + j]);
        }
    };
    fetch_gates(r0);

    int chunk_idx = 0;
    for (int rb = r0; rb < r1; rb += DC_C, ++chunk_idx) {
        const int Ce = min(DC_C, r1 - rb);
        const int slot = chunk_idx & 1;
        // ---- P1: causal conv + SiLU from the raw tile staged in shared memory by cp.async (the
        // copy for this chunk was issued while the previous chunk was being processed)
        cp_async_wait<0>();
        __syncthreads();
        // two adjacent channels per item (one 4-byte shared-memory load serves both), 8 rows per item
        for (int item = tid; item < (NCH / 2) * (DC_C / 8); item += DN_THREADS) {
            const int c = 2 * (item % (NCH / 2)), i0 = (item / (NCH / 2)) * 8;
            const float4 wa4 = *(const float4*)&cw[c * 4], wb4 = *(const float4*)&cw[c * 4 + 4];
            float* dst = (c < DK) ? Qs + c : (c < 2 * DK) ? Ks + (c - DK) : Us + (c - 2 * DK);
            const int ldd = (c < 2 * DK) ? LDK : DC_LDU;
            if (qk_pre && c < 2 * DK) {
                // already convolved and normalised by the pre-pass (fp16 holds exactly the ten mantissa bits the
                // TF32 products use): widen and store
#pragma unroll
                for (int i = i0; i < i0 + 8; ++i)
                    *(float2*)&dst[i * ldd] = __half22float2(*(const __half2*)&Xr[(i + 3) * NCH + c]);
                continue;
            }
            float2 x0 = __half22float2(*(const __half2*)&Xr[(i0 + 0) * NCH + c]);
            float2 x1 = __half22float2(*(const __half2*)&Xr[(i0 + 1) * NCH + c]);
            float2 x2 = __half22float2(*(const __half2*)&Xr[(i0 + 2) * NCH + c]);
#pragma unroll
            for (int i = i0; i < i0 + 8; ++i) {
                const float2 x3 = __half22float2(*(const __half2*)&Xr[(i + 3) * NCH + c]);
                const float a0 = x0.x * wa4.x + x1.x * wa4.y + x2.x * wa4.z + x3.x * wa4.w;
                const float a1 = x0.y * wb4.x + x1.y * wb4.y + x2.y * wb4.z + x3.y * wb4.w;
                *(float2*)&dst[i * ldd] = (i < Ce) ? make_float2(silu_fast(a0), silu_fast(a1)) : make_float2(0.f, 0.f);
                x0 = x1; x1 = x2; x2 = x3;
            }
        }
        if (tid < DC_C) {
            float gl = 0.f, beta = 0.f;
            if (tid < Ce) {
                const float a_in = a_pre, b_in = b_pre;
                float sp_ = a_in + dtb;
                gl = fmaxf(neg_expA * (sp_ > 20.f ? sp_ : log1pf(__expf(sp_))), -20.f);
                beta = sigmoid_f(b_in);
            }
            gs[tid] = gl;
            bs[tid] = beta;
            cl_ss[slot * DC_C + tid] = 0.f;
        }
        __syncthreads();
        if (rb + DC_C < r1) stage_raw(rb + DC_C);          // fly while this chunk is processed
        fetch_gates(rb + DC_C);
        // output gates of this chunk, needed only at its end
        float zf[DC_C / 8];
#pragma unroll
        for (int u = 0; u < DC_C / 8; ++u) {
            const int i = kr + 8 * u;
            zf[u] = (i < Ce) ? __half2float(p.proj[(size_t)(rb + i) * p.ld + p.off_z + j * DV + cb * DN_COLS + vcol]) : 0.f;
        }
        // ---- P2: L2-normalise q and k rows (stored rounded to TF32), running log-decay, state copy
        if (kr == 0) {
            // inclusive scan of the log-decays: DC_C / 32 per lane
            static_assert(DC_C == 32 || DC_C == 64, "chunk size");
            float a = gs[lane], b = DC_C > 32 ? gs[lane + DC_C - 32] : 0.f;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float ua = __shfl_up_sync(0xffffffffu, a, o), ub = __shfl_up_sync(0xffffffffu, b, o);
                if (lane >= o) { a += ua; b += ub; }
            }
            const float tot = __shfl_sync(0xffffffffu, a, 31);
            Gs[lane] = a;
            if (DC_C > 32) Gs[lane + DC_C - 32] = b + tot;
        }
#pragma unroll 1
        for (int ub = 0; ub < (qk_pre ? 0 : DC_C / 8); ub += 4) {
            // four rows at a time: their loads and the eight reductions overlap
            constexpr int PL = DK / 32;
            float qv[4][PL], kv[4][PL], qq[4], kk[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = kr + 8 * (ub + r);
                qq[r] = kk[r] = 0.f;
#pragma unroll
                for (int m = 0; m < PL; ++m) {
                    qv[r][m] = Qs[i * LDK + lane + 32 * m]; kv[r][m] = Ks[i * LDK + lane + 32 * m];
                    qq[r] += qv[r][m] * qv[r][m]; kk[r] += kv[r][m] * kv[r][m];
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    qq[r] += __shfl_xor_sync(0xffffffffu, qq[r], o);
                    kk[r] += __shfl_xor_sync(0xffffffffu, kk[r], o);
                }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = kr + 8 * (ub + r);
                const float iq = rsqrtf(qq[r] + 1e-6f) * qscale, ik = rsqrtf(kk[r] + 1e-6f);
#pragma unroll
                for (int m = 0; m < PL; ++m) {
                    Qs[i * LDK + lane + 32 * m] = tf32r(qv[r][m] * iq);
                    Ks[i * LDK + lane + 32 * m] = tf32r(kv[r][m] * ik);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < SPW; ++m) {
            const int mt = kr + 8 * m;
            if (mt < MT) {
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        S0t[(8 * n + 2 * t + (e & 1)) * LDK + 16 * mt + g + (e >> 1) * 8] = tf32r(S[m][n][e]);
            }
        }
        __syncthreads();
        // ---- P3: A = beta decay (K K^T) below the diagonal, W = decay (Q K^T) on and below it, in
        // 16x8 tiles of the lower triangle dealt round-robin to the warps.  Fragments come from
        // ldmatrix: one instruction per operand and k-step.
        constexpr int MB = DC_C / 16;                 // 16-row blocks of a chunk
        constexpr int NTW = (MB * 4) / 8;             // 8-column tiles of U / Y per warp in P4 and P6 (1 or 2)
        const int a_row = (lane & 7) + ((lane >> 3) & 1) * 8, a_col = (lane >> 4) * 4;       // A operand addressing
        const int b_row = (lane & 7) + (lane >> 4) * 8, b_col = ((lane >> 3) & 1) * 4;       // B operand, two 8-column tiles
        {
            for (int tile = kr; tile < MB * (MB + 1); tile += 8) {
                int mi = 0, ni = tile;                 // row block mi holds tiles ni = 0 .. 2 mi + 1
                while (ni >= 2 * mi + 2) { ni -= 2 * mi + 2; ++mi; }
                float kk[4] = {0.f, 0.f, 0.f, 0.f}, qk[4] = {0.f, 0.f, 0.f, 0.f};
                const float* ka = Ks + (16 * mi + a_row) * LDK + a_col;
                const float* qa = Qs + (16 * mi + a_row) * LDK + a_col;
                const float* kb = Ks + (8 * ni + (lane & 7)) * LDK + ((lane >> 3) & 1) * 4;   // x2: lanes 0-15 give the rows
#pragma unroll 4
                for (int k0 = 0; k0 < DK; k0 += 8) {
                    float fa[4], fq[4], fb[2];
                    ldsm4(fa, ka + k0); ldsm4(fq, qa + k0); ldsm2(fb, kb + k0);
                    mma_tf32(kk, fa[0], fa[1], fa[2], fa[3], fb[0], fb[1]);
                    mma_tf32(qk, fq[0], fq[1], fq[2], fq[3], fb[0], fb[1]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = 16 * mi + g + (e >> 1) * 8, jj = 8 * ni + 2 * t + (e & 1);
                    const float dec = (jj <= i) ? __expf(Gs[i] - Gs[jj]) : 0.f;
                    As[i * DC_LDA + jj] = (jj < i) ? bs[i] * dec * kk[e] : 0.f;
                    Ws[i * DC_LDA + jj] = tf32r(dec * qk[e]);
                }
            }
            // ---- P4: K S0 and Q S0; b = beta (v - exp(G) K S0) in place of v.  Warp w: row block
            // w % MB, column tiles NTW (w / MB) ...
            const int mi = kr % MB, nb = (kr / MB) * NTW;
            float ak[NTW][4], aq[NTW][4];
#pragma unroll
            for (int n = 0; n < NTW; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) ak[n][e] = aq[n][e] = 0.f;
            const float* ka = Ks + (16 * mi + a_row) * LDK + a_col;
            const float* qa = Qs + (16 * mi + a_row) * LDK + a_col;
            const float* sb4 = S0t + (8 * nb + b_row) * LDK + b_col;
            const float* sb2 = S0t + (8 * nb + (lane & 7)) * LDK + ((lane >> 3) & 1) * 4;
#pragma unroll 4
            for (int k0 = 0; k0 < DK; k0 += 8) {
                float fa[4], fq[4], fb[4];
                ldsm4(fa, ka + k0); ldsm4(fq, qa + k0);
                if constexpr (NTW == 2) {
                    ldsm4(fb, sb4 + k0);
                } else {
                    float f2[2];
                    ldsm2(f2, sb2 + k0);
                    fb[0] = f2[0]; fb[1] = f2[1]; fb[2] = fb[3] = 0.f;
                }
#pragma unroll
                for (int n = 0; n < NTW; ++n) {
                    mma_tf32(ak[n], fa[0], fa[1], fa[2], fa[3], fb[2 * n], fb[2 * n + 1]);
                    mma_tf32(aq[n], fq[0], fq[1], fq[2], fq[3], fb[2 * n], fb[2 * n + 1]);
                }
            }
#pragma unroll
            for (int n = 0; n < NTW; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = 16 * mi + g + (e >> 1) * 8, col = 8 * (nb + n) + 2 * t + (e & 1);
                    const float eg = __expf(Gs[i]);
                    Us[i * DC_LDU + col] = bs[i] * (Us[i * DC_LDU + col] - eg * ak[n][e]);
                    QSs[i * DN_COLS + col] = eg * aq[n][e];
                }
        }
        __syncthreads();
        // ---- P5: (I + A) U = B by forward substitution, 8 rows per block: every warp first removes
        // the contribution of all earlier blocks from its row, then warp 0 solves the 8x8 triangle
        // with one column per lane in registers
        for (int blk = 0; blk < DC_C / 8; ++blk) {
            const int i = 8 * blk + kr;
            float acc = Us[i * DC_LDU + vcol];
            for (int j0 = 0; j0 < 8 * blk; j0 += 8) {
                float av[8], uv[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) { av[q] = As[i * DC_LDA + j0 + q]; uv[q] = Us[(j0 + q) * DC_LDU + vcol]; }
#pragma unroll
                for (int q = 0; q < 8; ++q) acc = fmaf(-av[q], uv[q], acc);
            }
            Us[i * DC_LDU + vcol] = acc;
            __syncthreads();
            if (kr == 0) {
                float u[8];
#pragma unroll
                for (int a = 0; a < 8; ++a) u[a] = Us[(8 * blk + a) * DC_LDU + vcol];
#pragma unroll
                for (int a = 1; a < 8; ++a)
#pragma unroll
                    for (int b = 0; b < 8; ++b)
                        if (b < a) u[a] = fmaf(-As[(8 * blk + a) * DC_LDA + 8 * blk + b], u[b], u[a]);
#pragma unroll
                for (int a = 1; a < 8; ++a) Us[(8 * blk + a) * DC_LDU + vcol] = u[a];
            }
            __syncthreads();
        }
        // ---- P6: Y = exp(G) Q S0 + W U (W is zero above the diagonal), sum of squares per row
        {
            const int mi = kr % MB, nb = (kr / MB) * NTW;
            float y[NTW][4];
#pragma unroll
            for (int n = 0; n < NTW; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    y[n][e] = QSs[(16 * mi + g + (e >> 1) * 8) * DN_COLS + 8 * (nb + n) + 2 * t + (e & 1)];
            const float* wa = Ws + (16 * mi + a_row) * DC_LDA + a_col;
            for (int k0 = 0; k0 < 16 * (mi + 1); k0 += 8) {
                float fa[4];
                ldsm4(fa, wa + k0);
#pragma unroll
                for (int n = 0; n < NTW; ++n)
                    mma_tf32(y[n], fa[0], fa[1], fa[2], fa[3], tf32r(Us[(k0 + t) * DC_LDU + 8 * (nb + n) + g]),
                             tf32r(Us[(k0 + t + 4) * DC_LDU + 8 * (nb + n) + g]));
            }
            float s_lo = 0.f, s_hi = 0.f;
#pragma unroll
            for (int n = 0; n < NTW; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    Ys[(16 * mi + g + (e >> 1) * 8) * DN_COLS + 8 * (nb + n) + 2 * t + (e & 1)] = y[n][e];
                    if (e < 2) s_lo += y[n][e] * y[n][e]; else s_hi += y[n][e] * y[n][e];
                }
            s_lo += __shfl_xor_sync(0xffffffffu, s_lo, 1); s_lo += __shfl_xor_sync(0xffffffffu, s_lo, 2);
            s_hi += __shfl_xor_sync(0xffffffffu, s_hi, 1); s_hi += __shfl_xor_sync(0xffffffffu, s_hi, 2);
            if (t == 0) {
                atomicAdd(&cl_ss[slot * DC_C + 16 * mi + g], s_lo);
                atomicAdd(&cl_ss[slot * DC_C + 16 * mi + g + 8], s_hi);
            }
        }
        // ---- P7: S' = exp(G_C) S0 + K^T (exp(G_C - G) U), accumulated into the register fragments
        {
            const float gC = Gs[DC_C - 1];
            const float egC = __expf(gC);
#pragma unroll
            for (int m = 0; m < SPW; ++m)
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) S[m][n][e] *= egC;
            for (int k0 = 0; k0 < DC_C; k0 += 8) {
                const float tl0 = __expf(gC - Gs[k0 + t]), tl1 = __expf(gC - Gs[k0 + t + 4]);
                float b0[4], b1[4];
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    b0[n] = tf32r(Us[(k0 + t) * DC_LDU + 8 * n + g] * tl0);
                    b1[n] = tf32r(Us[(k0 + t + 4) * DC_LDU + 8 * n + g] * tl1);
                }
#pragma unroll
                for (int m = 0; m < SPW; ++m) {
                    const int mt = kr + 8 * m;
                    if (mt < MT) {
                        // A = K^T: element (dk row, chunk row) = Ks[chunk row][dk row]
                        const float* kt = Ks + (k0 + t) * LDK + 16 * mt + g;
                        const float a0 = kt[0], a1 = kt[8], a2 = kt[4 * LDK], a3 = kt[4 * LDK + 8];
#pragma unroll
                        for (int n = 0; n < 4; ++n) mma_tf32(S[m][n], a0, a1, a2, a3, b0[n], b1[n]);
                    }
                }
            }
        }
        cluster.sync();
        // ---- gated RMSNorm across the head's column blocks, output.  The warp's DC_C/8 rows x CB
        // peers are read from distributed shared memory by that many lanes at once, and the gate values are
        // loaded before anything is stored.
        {
            float v = 0.f;
            if (lane < (DC_C / 8) * CB) v = cluster.map_shared_rank(cl_ss, lane % CB)[slot * DC_C + kr + 8 * (lane / CB)];
#pragma unroll
            for (int o = CB / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
#pragma unroll
            for (int u = 0; u < DC_C / 8; ++u) {
                const int i = kr + 8 * u;
                const float tot = __shfl_sync(0xffffffffu, v, u * CB);
                if (i < Ce) {
                    const float o = Ys[i * DN_COLS + vcol] * rsqrtf(tot / (float)DV + p.eps) * nw * silu_fast(zf[u]);
                    p.out[(size_t)(rb + i) * p.ldo + j * DV + cb * DN_COLS + vcol] = __float2half(o);
                }
            }
        }
        __syncthreads();
    }
    cluster.sync();
    if (!p.commit) return;
#pragma unroll
    for (int m = 0; m < SPW; ++m) {
        const int mt = kr + 8 * m;
        if (mt < MT) {
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                *(float2*)(sp + (size_t)(16 * mt + g) * DV + 8 * n + 2 * t) = make_float2(S[m][n][0], S[m][n][1]);
                *(float2*)(sp + (size_t)(16 * mt + g + 8) * DV + 8 * n + 2 * t) = make_float2(S[m][n][2], S[m][n][3]);
            }
        }
    }
    // last three raw conv inputs (older history shifts in when the sequence was shorter than 3 rows)
    for (int c = tid; c < NCH; c += DN_THREADS) {
        const int col = proj_col(c);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int ri = r1 - 3 + q;
            float x = (ri >= r0) ? __half2float(p.proj[(size_t)ri * p.ld + col]) : hist[c * 3 + (ri - r0 + 3)];
            my_hist[c * 3 + q] = __float2half(x);
        }
    }
}

// ---------------------------------------------------------------------------
// Pre-pass of the chunked scan: causal conv + SiLU + L2 norm of the q and k channels of every row, once
// per key head and fully parallel over the rows (the scan kernel would otherwise redo it in each of the
// dv/32 column CTAs of each of the nv/nk value heads that share a key head, on its sequential path).
// Output fp16 [rows][2 * nk * DK]: q (scaled by 1/sqrt(DK)) | k.  A warp owns a head's q or k over QP_ROWS rows: a lane has
// DK / 32 adjacent channels, so rows are read and written in pieces of 256 bytes a warp and the norm stays inside the warp.
// Bound: the rows' bytes.  (A thread with one channel of 16 rows: 12 us for 512 rows of 16 heads, 75 us for 3001; now 8 and 25.)
// grid = (row blocks of QP_ROWS, 2 nk / 8), eight warps.
// ---------------------------------------------------------------------------
#define QP_ROWS 8
template <int DK>
__global__ void __launch_bounds__(256) deltanet_qk_prep_kernel(const DeltaParams p, __half* __restrict__ qk_pre, int ld_qk,
                                                               int cb_copies, int nch) {
    constexpr int CH = DK / 32;                    // channels of a lane: 4 or 2
    struct alignas(2 * CH) Chans { __half v[CH]; };
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, unit = blockIdx.y * 8 + (threadIdx.x >> 5);       // q heads, then k heads
    const int r0 = p.seq_rows[0], r1 = p.seq_rows[1];
    const int rb = r0 + blockIdx.x * QP_ROWS;
    if (rb >= r1 || unit >= 2 * p.nk) return;
    const int seq = p.rows[r0].seq;
    const bool is_q = unit < p.nk;
    const int kh = is_q ? unit : unit - p.nk, c = lane * CH;
    const int col = (is_q ? p.off_q : p.off_k) + kh * DK + c;
    float w[CH][4];
#pragma unroll
    for (int e = 0; e < CH; ++e)
#pragma unroll
        for (int q = 0; q < 4; ++q) w[e][q] = __half2float(p.conv_w[(size_t)(unit * DK + c + e) * 4 + q]);
    // rows before the sequence start come from the saved history of the first value head of this key head
    const __half* hist = p.conv_state + ((((size_t)seq * p.nv + kh * (p.nv / p.nk)) * cb_copies) * nch + (is_q ? 0 : DK) + c) * 3;
    const bool whole = ((p.ld | col) & (CH - 1)) == 0 && ((uintptr_t)p.proj & (2 * CH - 1)) == 0;
    // all rows are requested before the first is looked at (rows outside the launch read one inside and are replaced)
    Chans v[QP_ROWS + 3];
    if (whole) {
#pragma unroll
        for (int i = 0; i < QP_ROWS + 3; ++i) v[i] = *(const Chans*)(p.proj + (size_t)min(max(rb - 3 + i, r0), r1 - 1) * p.ld + col);
    } else {
#pragma unroll
        for (int i = 0; i < QP_ROWS + 3; ++i)
#pragma unroll
            for (int e = 0; e < CH; ++e) v[i].v[e] = p.proj[(size_t)min(max(rb - 3 + i, r0), r1 - 1) * p.ld + col + e];
    }
    if (rb == r0) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int e = 0; e < CH; ++e) v[i].v[e] = hist[e * 3 + i];
    }
    float x[QP_ROWS + 3][CH];
#pragma unroll
    for (int i = 0; i < QP_ROWS + 3; ++i)
#pragma unroll
        for (int e = 0; e < CH; ++e) x[i][e] = __half2float(v[i].v[e]);
    const float qscale = is_q ? rsqrtf((float)DK) : 1.f;
#pragma unroll
    for (int i = 0; i < QP_ROWS; ++i) {
        float y[CH], ss = 0.f;
#pragma unroll
        for (int e = 0; e < CH; ++e) {
            y[e] = silu_fast(x[i][e] * w[e][0] + x[i + 1][e] * w[e][1] + x[i + 2][e] * w[e][2] + x[i + 3][e] * w[e][3]);
            ss += y[e] * y[e];
        }
        const float inv = rsqrtf(warp_sum(ss) + 1e-6f) * qscale;
        if (rb + i >= r1) break;
        Chans o;
#pragma unroll
        for (int e = 0; e < CH; ++e) o.v[e] = __float2half_rn(y[e] * inv);
        *(Chans*)(qk_pre + (size_t)(rb - r0 + i) * ld_qk + unit * DK + c) = o;
    }
}

// ---------------------------------------------------------------------------
// The scan of one prompt, in three parts.  With T = (I + A)^-1 the update vectors of a chunk are
//     U = T (beta (V - exp(G) K S0)) = U0 - Wt S0,     U0 = T diag(beta) V,   Wt = T diag(beta exp(G)) K,
// and U0, Wt and W do not depend on the state.  So a first kernel forms them for every (value head, chunk) side by side
// (deltanet_tw_prep_kernel), and what is left to the serial walk over the chunks is two dependent products a chunk:
// [Wt; Q] S0, then W U and K^T U (deltanet_scan_kernel).  The raw outputs go back into U0's place; a third kernel
// norms, gates and rounds them (deltanet_scan_out_kernel), which also keeps the sum over a head's columns, and with it
// the cluster, out of the walk.
//
// Per (value head, chunk) the work buffer holds Wt [32][DK] | U0, later Y [32][DV] | W [32][32] | exp(G) [32] |
// exp(G_C - G) [32] | exp(G_C).
// ---------------------------------------------------------------------------
#define DC_GATES (2 * DC_C + 4)
template <int DK, int DV> struct ScanBlock {
    static constexpr int U0 = DC_C * DK, W = U0 + DC_C * DV, GATES = W + DC_C * DC_C, FLOATS = GATES + DC_GATES;
};

// x = hi + lo with hi rounded to a TF32 value (as tf32r does; an addition and a mask take fewer issue slots than the
// conversion).  At most 13 bits are left for lo, of which the tensor core reads 11: 2^-23 of x is cut off at most.
__device__ __forceinline__ void split_tf32(float x, float& hi, float& lo) {
    hi = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
    lo = x - hi;
}
__device__ __forceinline__ void ldsm4_h(uint32_t (&r)[4], const __half* row_ptr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(row_ptr)));
}
__device__ __forceinline__ void ldsm4_ht(uint32_t (&r)[4], const __half* row_ptr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(row_ptr)));
}
__device__ __forceinline__ float2 h2f(uint32_t x) { return __half22float2(*(const __half2*)&x); }

// Everything of a chunk that does not depend on the state: the gates, A = beta decay (K K^T) below the diagonal,
// W = decay (Q K^T) on and below it, T = (I + A)^-1 (forward substitution on the two 16 x 16 diagonal triangles, one column per
// lane, and two products for the block below them), the convolved values V, and with them U0 and Wt.  T enters its products as hi + lo TF32 parts (and V too; K is
// fp16), so they keep fp32 accuracy.  grid = (chunks, value heads), 256 threads.
template <int DK, int DV>
__global__ void __launch_bounds__(DN_THREADS) deltanet_tw_prep_kernel(const DeltaParams p, const __half* __restrict__ ab, int ld_ab,
                                                                      const __half* __restrict__ qk_pre, int ld_qk,
                                                                      float* __restrict__ tw, int n_chunks) {
    static_assert(DC_C == 32, "a warp has the chunk's rows, half of one a column of a triangle each");
    constexpr int LDK = DC_LDK(DK), LDV = DV + 8;
    constexpr int MB = DC_C / 16;
    extern __shared__ __align__(16) float psm[];
    pdl_launch_dependents();
    pdl_wait();
    float* Qs = psm;                          // [C][LDK]
    float* Ks = Qs + DC_C * LDK;
    float* Vs = Ks + DC_C * LDK;              // [C][LDV]
    float* As = Vs + DC_C * LDV;              // [C][LDA]
    float* Ws = As + DC_C * DC_LDA;
    float* Ts = Ws + DC_C * DC_LDA;
    float* Gs = Ts + DC_C * DC_LDA;           // [C]
    float* bs = Gs + DC_C;
    const int ci = blockIdx.x, j = blockIdx.y, kh = j / (p.nv / p.nk);
    const int tid = threadIdx.x, lane = tid & 31, kr = tid >> 5, g = lane >> 2, t = lane & 3;
    const int r0 = p.seq_rows[0], r1 = p.seq_rows[1];
    const int rb = r0 + ci * DC_C;
    if (rb >= r1) return;
    const int Ce = min(DC_C, r1 - rb), seq = p.rows[r0].seq;
    // everything is requested before the first value is looked at: loads behind conditions, each with its conversion, were
    // taken one after the other, which was half of this kernel's time (14 600 of 30 000 clocks)
    constexpr int NQK = DC_C * (DK / 8) * 2 / DN_THREADS, NV = DV * (DC_C / 8) / DN_THREADS;
    static_assert(NQK * DN_THREADS == DC_C * (DK / 8) * 2 && NV * DN_THREADS == DV * (DC_C / 8), "whole turns of the threads");
    uint4 qk[NQK];
    __half vx[NV][11], vw[NV][4];
#pragma unroll
    for (int q = 0; q < NQK; ++q) {
        const int idx = tid + q * DN_THREADS, which = idx / (DC_C * (DK / 8)), rem = idx % (DC_C * (DK / 8));
        const int row = rem / (DK / 8), c = (rem % (DK / 8)) * 8;
        qk[q] = *(const uint4*)(qk_pre + (size_t)(rb - r0 + min(row, Ce - 1)) * ld_qk + (which ? p.nk * DK : 0) + kh * DK + c);
    }
    // values: causal convolution + SiLU of a channel over a run of rows; rows before the sequence come from the history
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const int idx = tid + q * DN_THREADS, c = idx % DV, i0 = idx / DV * 8;
        const __half* col = p.proj + p.off_v + j * DV + c;
        const __half* w = p.conv_w + (size_t)(2 * p.nk * DK + j * DV + c) * 4;
#pragma unroll
        for (int i = 0; i < 11; ++i) vx[q][i] = col[(size_t)min(max(rb + i0 - 3 + i, r0), r1 - 1) * p.ld];
#pragma unroll
        for (int i = 0; i < 4; ++i) vw[q][i] = w[i];
        if (ci == 0 && i0 == 0) {
            const __half* hist = p.conv_state + ((((size_t)seq * p.nv + j) * (DV / DN_COLS) + c / DN_COLS) * (2 * DK + DN_COLS) + 2 * DK + c % DN_COLS) * 3;
#pragma unroll
            for (int i = 0; i < 3; ++i) vx[q][i] = hist[i];
        }
    }
    __half ga = __float2half(0.f), gb = ga, g_bias = ga;
    float g_log = 0.f;
    if (tid < DC_C) {
        const __half* abr = ab + (size_t)(rb + min(tid, Ce - 1)) * ld_ab;
        ga = abr[j]; gb = abr[p.nv + j]; g_bias = p.dt_bias[j]; g_log = p.A_log[j];
    }
#pragma unroll
    for (int q = 0; q < NQK; ++q) {
        const int idx = tid + q * DN_THREADS, which = idx / (DC_C * (DK / 8)), rem = idx % (DC_C * (DK / 8));
        const int row = rem / (DK / 8), c = (rem % (DK / 8)) * 8;
        const __half2* h2 = (const __half2*)&qk[q];
        float f[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) { const float2 v = __half22float2(h2[e]); f[2 * e] = row < Ce ? v.x : 0.f; f[2 * e + 1] = row < Ce ? v.y : 0.f; }
        float* dst = (which ? Ks : Qs) + row * LDK + c;
        *(float4*)dst = make_float4(f[0], f[1], f[2], f[3]);
        *(float4*)(dst + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const int idx = tid + q * DN_THREADS, c = idx % DV, i0 = idx / DV * 8;
        float x[11], w[4];
#pragma unroll
        for (int i = 0; i < 11; ++i) x[i] = __half2float(vx[q][i]);
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = __half2float(vw[q][i]);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            Vs[(i0 + i) * LDV + c] = i0 + i < Ce ? silu_fast(x[i] * w[0] + x[i + 1] * w[1] + x[i + 2] * w[2] + x[i + 3] * w[3]) : 0.f;
    }
    if (tid < DC_C) {
        float gl = 0.f, beta = 0.f;
        if (tid < Ce) {
            const float sp_ = __half2float(ga) + __half2float(g_bias);
            gl = fmaxf(-__expf(g_log) * (sp_ > 20.f ? sp_ : log1pf(__expf(sp_))), -20.f);
            beta = sigmoid_f(__half2float(gb));
        }
        bs[tid] = beta;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {           // (the first warp has the chunk's rows)
            const float ua = __shfl_up_sync(0xffffffffu, gl, o);
            if (lane >= o) gl += ua;
        }
        Gs[tid] = gl;
    }
    __syncthreads();
    {
        const int a_row = (lane & 7) + ((lane >> 3) & 1) * 8, a_col = (lane >> 4) * 4;
        for (int tile = kr; tile < MB * (MB + 1); tile += 8) {
            int mi = 0, ni = tile;                 // row block mi holds tiles ni = 0 .. 2 mi + 1
            while (ni >= 2 * mi + 2) { ni -= 2 * mi + 2; ++mi; }
            float kk[4] = {0.f, 0.f, 0.f, 0.f}, qk[4] = {0.f, 0.f, 0.f, 0.f};
            const float* ka = Ks + (16 * mi + a_row) * LDK + a_col;
            const float* qa = Qs + (16 * mi + a_row) * LDK + a_col;
            const float* kb = Ks + (8 * ni + (lane & 7)) * LDK + ((lane >> 3) & 1) * 4;
#pragma unroll 4
            for (int k0 = 0; k0 < DK; k0 += 8) {
                float fa[4], fq[4], fb[2];
                ldsm4(fa, ka + k0); ldsm4(fq, qa + k0); ldsm2(fb, kb + k0);
                mma_tf32(kk, fa[0], fa[1], fa[2], fa[3], fb[0], fb[1]);
                mma_tf32(qk, fq[0], fq[1], fq[2], fq[3], fb[0], fb[1]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = 16 * mi + g + (e >> 1) * 8, jj = 8 * ni + 2 * t + (e & 1);
                const float dec = (jj <= i) ? __expf(Gs[i] - Gs[jj]) : 0.f;
                As[i * DC_LDA + jj] = (jj < i) ? bs[i] * dec * kk[e] : 0.f;
                Ws[i * DC_LDA + jj] = tf32r(dec * qk[e]);
            }
        }
        // tiles above the diagonal were not visited: they are zero
        for (int idx = tid; idx < DC_C * DC_C; idx += DN_THREADS) {
            const int i = idx / DC_C, jj = idx % DC_C;
            if ((jj >> 3) > ((i >> 4) * 2 + 1)) { As[i * DC_LDA + jj] = 0.f; Ws[i * DC_LDA + jj] = 0.f; }
        }
    }
    __syncthreads();
    // T = [T1 0; -T2 A21 T1  T2] with T1, T2 the inverses of the diagonal 16 x 16 triangles of I + A: a warp forms one by
    // forward substitution, a column per lane (t_i = [i == c] - sum_{j < i} A_ij t_j); then all threads two 16 x 16 products.
    // (One warp over all 32 rows took 3500-4200 clocks, while the others waited.)
    constexpr int HC = DC_C / 2;
    if (kr < 2) {
        const float* Ad = As + kr * (HC * DC_LDA + HC);
        float* Td = Ts + kr * (HC * DC_LDA + HC);
        const int c = lane & (HC - 1);
        float tc[HC];
#pragma unroll
        for (int i = 0; i < HC; ++i) {
            float v = (i == c) ? 1.f : 0.f;
#pragma unroll
            for (int jj = 0; jj < HC; ++jj)
                if (jj < i) v = fmaf(-Ad[i * DC_LDA + jj], tc[jj], v);
            tc[i] = v;
            if (lane < HC) Td[i * DC_LDA + c] = v;
        }
    }
    __syncthreads();
    const int hr = tid / HC, hc = tid % HC;                    // 256 threads: an element each
    {
        float v = 0.f;                                         // A21 T1, kept where T is zero
#pragma unroll
        for (int k = 0; k < HC; ++k) v = fmaf(As[(HC + hr) * DC_LDA + k], Ts[k * DC_LDA + hc], v);
        Ts[hr * DC_LDA + HC + hc] = v;
    }
    __syncthreads();
    float t21 = 0.f;
#pragma unroll
    for (int k = 0; k < HC; ++k) t21 = fmaf(-Ts[(HC + hr) * DC_LDA + HC + k], Ts[k * DC_LDA + HC + hc], t21);
    __syncthreads();
    Ts[(HC + hr) * DC_LDA + hc] = t21;
    Ts[hr * DC_LDA + HC + hc] = 0.f;
    __syncthreads();
    typedef ScanBlock<DK, DV> B;
    float* dst = tw + ((size_t)j * n_chunks + ci) * B::FLOATS;
    for (int idx = tid; idx < DC_C * DC_C; idx += DN_THREADS) dst[B::W + idx] = Ws[(idx / DC_C) * DC_LDA + idx % DC_C];
    if (tid < DC_C) {
        dst[B::GATES + tid] = __expf(Gs[tid]);
        dst[B::GATES + DC_C + tid] = __expf(Gs[DC_C - 1] - Gs[tid]);
        if (tid == 0) dst[B::GATES + 2 * DC_C] = __expf(Gs[DC_C - 1]);
    }
    // ---- Wt = (T diag(beta exp(G))) K and U0 = (T diag(beta)) V: 16 x 8 tiles, T is zero above the diagonal
    // (a warp keeps to one row tile, so T's fragments are split once per product)
    const int mi = kr % MB;
#pragma unroll
    for (int kind = 0; kind < 2; ++kind) {
        const bool is_k = kind == 0;
        const float* src = is_k ? Ks + g : Vs + g;
        const int lds = is_k ? LDK : LDV, ldo = is_k ? DK : DV;
        float* o = dst + (is_k ? 0 : B::U0) + 2 * t;
        float hi[DC_C / 8][4], lo[DC_C / 8][4];
#pragma unroll
        for (int k8 = 0; k8 < DC_C / 8; ++k8)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int k = 8 * k8 + t + 4 * (e >> 1);
                split_tf32(Ts[(16 * mi + g + 8 * (e & 1)) * DC_LDA + k] * bs[k] * (is_k ? __expf(Gs[k]) : 1.f), hi[k8][e], lo[k8][e]);
            }
        for (int n0 = kr / MB * 8; n0 < ldo; n0 += DN_THREADS / 32 / MB * 8) {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k8 = 0; k8 < DC_C / 8; ++k8) {
                if (8 * k8 >= 16 * (mi + 1)) break;
                float h0, l0, h1, l1;
                split_tf32(src[n0 + (8 * k8 + t) * lds], h0, l0);
                split_tf32(src[n0 + (8 * k8 + t + 4) * lds], h1, l1);
                mma_tf32(acc, lo[k8][0], lo[k8][1], lo[k8][2], lo[k8][3], h0, h1);
                if (!is_k) mma_tf32(acc, hi[k8][0], hi[k8][1], hi[k8][2], hi[k8][3], l0, l1);      // (K is exact)
                mma_tf32(acc, hi[k8][0], hi[k8][1], hi[k8][2], hi[k8][3], h0, h1);
            }
            *(float2*)(o + (16 * mi + g) * ldo + n0) = make_float2(acc[0], acc[1]);
            *(float2*)(o + (16 * mi + g + 8) * ldo + n0) = make_float2(acc[2], acc[3]);
        }
    }
}

// The walk over the chunks.  A CTA owns COLS columns of a value head's state: as accumulator fragments in registers (warp w:
// rows 16 w ..) and, TF32-rounded and transposed, as the B operand in shared memory.  Two barriers a chunk:
//   A  warp (m, n) forms its 16 x 8 tiles (one, or of 64 columns two) of Wt S0 (Wt as hi + lo) and Q S0, and writes U, twice (plain, and times
//      exp(G_C - G) for the state), as a transposed B operand;
//   B  the same warp finishes its tile of Y = exp(G) Q S0 + W U, and every warp updates its rows of the state.
// The operands of the next chunk travel meanwhile (cp.async, two stages).  The order of k inside a product is free: a
// 16-k block is taken as (2t, 2t + 1) and (8 + 2t, 9 + 2t), which is what ldmatrix gives of fp16 rows and one 8-byte
// load of fp32 rows.  Bound: the latency of this chain.  Measured (48 value heads of 128, 512 rows):
// 53 us, and 26 + 8 us for the parts before and behind it; one kernel with nine barriers a chunk took 144 + 16 us.
// COLS: two CTAs on an SM hinder one another (1.7 us a chunk alone, 3.8 both), so the grid has at most one for each SM where
// that can be: 32 columns up to 37 value heads, 64 up to 74 (their second tile takes the loaded Wt and Q again), else
// 32 and two CTAs an SM.  48 heads, 512 rows: 32 columns 60 us, 64 53; 32 heads, 3001 rows: two CTAs on some SMs, because the
// first SMs that the kernel before left took two, 360 us, one on each 218.
#define SC_LDH(D) ((D) + 8)      // halfs: 16-byte rows of 8 adjacent lanes meet no bank twice
#define SC_LDF(D) ((D) + 8)      // floats: the 8-byte reads of a half warp neither
template <int DK>
struct ScanStage {
    __half q[DC_C][SC_LDH(DK)], k[DC_C][SC_LDH(DK)];
    float wt[DC_C][SC_LDF(DK)], w[DC_C][SC_LDF(DC_C)], gates[DC_GATES];
};
template <int DK, int COLS>
struct ScanSmem {
    ScanStage<DK> st[2];
    float s0[COLS][SC_LDF(DK)], u[COLS][SC_LDF(DC_C)], ut[COLS][SC_LDF(DC_C)];
};

template <int DK, int DV, int COLS>
__global__ void __launch_bounds__(DN_THREADS, COLS == 32 ? 2 : 1) deltanet_scan_kernel(const DeltaParams p, const __half* __restrict__ qk_pre, int ld_qk,
                                                                     float* __restrict__ tw, int n_chunks) {
    typedef ScanBlock<DK, DV> B;
    constexpr int MT = DK / 16;                   // warps that own 16 rows of the state
    constexpr int NT = COLS / 32, NS = COLS / 8;  // column tiles of a warp in A (32 columns apart), of the state
    static_assert(DC_C == 32 && COLS % 32 == 0 && MT <= 8, "eight warps: two row tiles by four column tiles");
    extern __shared__ __align__(16) float dsm[];
    ScanSmem<DK, COLS>& sm = *(ScanSmem<DK, COLS>*)dsm;
    pdl_launch_dependents();
    if (!p.older) pdl_wait();
    const int cb = blockIdx.x, j = blockIdx.y, kh = j / (p.nv / p.nk);
    const int tid = threadIdx.x, lane = tid & 31, kr = tid >> 5, g = lane >> 2, t = lane & 3;
    const int r0 = p.seq_rows[0], r1 = p.seq_rows[1];
    if (r0 >= r1) return;
    const int seq = p.rows[r0].seq, chunks = min((r1 - r0 + DC_C - 1) / DC_C, n_chunks);
    float* blocks = tw + (size_t)j * n_chunks * B::FLOATS;

    auto stage = [&](int ci) {
        ScanStage<DK>& s = sm.st[ci & 1];
        const float* src = blocks + (size_t)ci * B::FLOATS;
        for (int i = tid; i < DC_C * (DK / 8) * 2; i += DN_THREADS) {
            const int which = i / (DC_C * (DK / 8)), row = i / (DK / 8) % DC_C, c = i % (DK / 8) * 8, ri = ci * DC_C + row;
            __half* d = which ? &s.k[row][c] : &s.q[row][c];
            if (r0 + ri < r1) cp_async16(d, qk_pre + (size_t)ri * ld_qk + (which ? p.nk * DK : 0) + kh * DK + c);
            else *(uint4*)d = make_uint4(0u, 0u, 0u, 0u);
        }
        for (int i = tid; i < DC_C * (DK / 4); i += DN_THREADS) cp_async16(&s.wt[i / (DK / 4)][i % (DK / 4) * 4], src + 4 * i);
        for (int i = tid; i < DC_C * (DC_C / 4); i += DN_THREADS) cp_async16(&s.w[i / (DC_C / 4)][i % (DC_C / 4) * 4], src + B::W + 4 * i);
        if (tid < DC_GATES / 4) cp_async16(&s.gates[4 * tid], src + B::GATES + 4 * tid);
        cp_async_commit();
    };
    // this lane's elements of its 16 x 8 tiles of U0 (and later Y)
    const int mi = kr & 1, ni = kr >> 1;
    const size_t u0_off = (size_t)B::U0 + (size_t)(16 * mi + g) * DV + cb * COLS + 8 * ni + 2 * t;
    float2 u0[NT][2], u0n[NT][2] = {};
    auto load_u0 = [&](int ci) {
        const float* src = blocks + (size_t)ci * B::FLOATS + u0_off;
#pragma unroll
        for (int c = 0; c < NT; ++c) {
            u0n[c][0] = *(const float2*)(src + 32 * c);
            u0n[c][1] = *(const float2*)(src + 32 * c + 8 * DV);
        }
    };
    float S[NS][4];
    float* sp = p.state + (((size_t)seq * p.nv + j) * DK) * DV + cb * COLS;
    auto put_s0 = [&]() {
        if (kr < MT) {
#pragma unroll
            for (int n = 0; n < NS; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) sm.s0[8 * n + 2 * t + (e & 1)][16 * kr + g + 8 * (e >> 1)] = tf32r(S[n][e]);
        }
    };
    if (kr < MT) {
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            const float2 lo = *(const float2*)(sp + (size_t)(16 * kr + g) * DV + 8 * n + 2 * t);
            const float2 hi = *(const float2*)(sp + (size_t)(16 * kr + g + 8) * DV + 8 * n + 2 * t);
            S[n][0] = lo.x; S[n][1] = lo.y; S[n][2] = hi.x; S[n][3] = hi.y;
        }
    }
    pdl_wait();
    stage(0);
    load_u0(0);
    put_s0();
    const int a_row = lane & 15, a_col = (lane >> 4) * 8;                              // fp16 A operand (ldmatrix)
    const int kt_row = (lane & 7) + (lane & 8), kt_col = (lane >> 4) * 8;              // its transpose: chunk rows x state rows
    for (int ci = 0; ci < chunks; ++ci) {
        cp_async_wait<0>();
        __syncthreads();                          // the chunk's operands and S0 are in place; everyone left the chunk before
        if (ci + 1 < chunks) stage(ci + 1);
#pragma unroll
        for (int c = 0; c < NT; ++c) { u0[c][0] = u0n[c][0]; u0[c][1] = u0n[c][1]; }
        if (ci + 1 < chunks) load_u0(ci + 1);
        const ScanStage<DK>& s = sm.st[ci & 1];
        // ---- A
        float wh[NT][4] = {}, wl[NT][4] = {}, y[NT][4] = {};
        {
            const float* wr = &s.wt[16 * mi + g][2 * t];
            const float* br = &sm.s0[8 * ni + g][2 * t];
            const __half* qr = &s.q[16 * mi + a_row][a_col];
#pragma unroll
            for (int k0 = 0; k0 < DK; k0 += 16) {
                uint32_t q[4];
                ldsm4_h(q, qr + k0);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 x = *(const float2*)(wr + k0 + 8 * h), z = *(const float2*)(wr + 8 * SC_LDF(DK) + k0 + 8 * h);
                    const float2 qa = h2f(q[2 * h]), qb = h2f(q[2 * h + 1]);
                    float hi[4], lo[4];
                    split_tf32(x.x, hi[0], lo[0]); split_tf32(z.x, hi[1], lo[1]);
                    split_tf32(x.y, hi[2], lo[2]); split_tf32(z.y, hi[3], lo[3]);
#pragma unroll
                    for (int c = 0; c < NT; ++c) {
                        const float2 b = *(const float2*)(br + 32 * c * SC_LDF(DK) + k0 + 8 * h);
                        mma_tf32(wh[c], hi[0], hi[1], hi[2], hi[3], b.x, b.y);
                        mma_tf32(wl[c], lo[0], lo[1], lo[2], lo[3], b.x, b.y);
                        mma_tf32(y[c], qa.x, qb.x, qa.y, qb.y, b.x, b.y);
                    }
                }
            }
        }
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = 16 * mi + g + 8 * (e >> 1), c = 32 * n + 8 * ni + 2 * t + (e & 1);
                const float u = ((e & 2) ? ((e & 1) ? u0[n][1].y : u0[n][1].x) : ((e & 1) ? u0[n][0].y : u0[n][0].x)) - (wh[n][e] + wl[n][e]);
                sm.u[c][i] = tf32r(u);
                sm.ut[c][i] = tf32r(u * s.gates[DC_C + i]);
                y[n][e] *= s.gates[i];
            }
        __syncthreads();
        // ---- B: Y
        {
            const float* wr = &s.w[16 * mi + g][2 * t];
            const float* br = &sm.u[8 * ni + g][2 * t];
#pragma unroll
            for (int k0 = 0; k0 < DC_C; k0 += 8) {
                if (k0 >= 16 * (mi + 1)) break;   // (W is zero above the diagonal)
                const float2 x = *(const float2*)(wr + k0), z = *(const float2*)(wr + 8 * SC_LDF(DC_C) + k0);
#pragma unroll
                for (int c = 0; c < NT; ++c) {
                    const float2 b = *(const float2*)(br + 32 * c * SC_LDF(DC_C) + k0);
                    mma_tf32(y[c], x.x, z.x, x.y, z.y, b.x, b.y);
                }
            }
            float* dst = blocks + (size_t)ci * B::FLOATS + u0_off;
#pragma unroll
            for (int c = 0; c < NT; ++c) {
                *(float2*)(dst + 32 * c) = make_float2(y[c][0], y[c][1]);
                *(float2*)(dst + 32 * c + 8 * DV) = make_float2(y[c][2], y[c][3]);
            }
        }
        // ---- B: S' = exp(G_C) S0 + K^T (exp(G_C - G) U)
        if (kr < MT) {
            const float egC = s.gates[2 * DC_C];
#pragma unroll
            for (int n = 0; n < NS; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[n][e] *= egC;
#pragma unroll
            for (int k0 = 0; k0 < DC_C; k0 += 16) {
                uint32_t kt[4];                   // chunk rows k0 + 2t, state row g | k0 + 8 + 2t, g | k0 + 2t, g + 8 | k0 + 8 + 2t, g + 8
                ldsm4_ht(kt, &s.k[k0 + kt_row][16 * kr + kt_col]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 lo = h2f(kt[h]), hi = h2f(kt[2 + h]);
#pragma unroll
                    for (int n = 0; n < NS; ++n) {
                        const float2 b = *(const float2*)&sm.ut[8 * n + g][k0 + 8 * h + 2 * t];
                        mma_tf32(S[n], lo.x, hi.x, lo.y, hi.y, b.x, b.y);
                    }
                }
            }
        }
        put_s0();                                 // (every warp read S0 before the second barrier)
    }
    if (!p.commit) return;
    if (kr < MT) {
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            *(float2*)(sp + (size_t)(16 * kr + g) * DV + 8 * n + 2 * t) = make_float2(S[n][0], S[n][1]);
            *(float2*)(sp + (size_t)(16 * kr + g + 8) * DV + 8 * n + 2 * t) = make_float2(S[n][2], S[n][3]);
        }
    }
}

// Gated RMSNorm of the raw outputs, one warp per (row, value head); the CTAs behind the rows store the last three raw
// convolution inputs of every channel (older history shifts in when the prompt was shorter than that).
template <int DK, int DV>
__global__ void __launch_bounds__(DN_THREADS) deltanet_scan_out_kernel(const DeltaParams p, const float* __restrict__ tw, int n_chunks, int row_ctas) {
    typedef ScanBlock<DK, DV> B;
    constexpr int PL = DV / 32;
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31;
    const int r0 = p.seq_rows[0], r1 = p.seq_rows[1];
    if (r0 >= r1) return;
    if ((int)blockIdx.x >= row_ctas) {
        if (!p.commit) return;
        constexpr int NCH = 2 * DK + DN_COLS, CB = DV / DN_COLS;
        const int hb = blockIdx.x - row_ctas, j = hb / CB, cb = hb % CB, kh = j / (p.nv / p.nk);
        __half* hist = p.conv_state + ((((size_t)p.rows[r0].seq * p.nv + j) * CB + cb) * NCH) * 3;
        for (int c = tid; c < NCH; c += DN_THREADS) {
            const int col = c < DK ? p.off_q + kh * DK + c : (c < 2 * DK ? p.off_k + kh * DK + c - DK : p.off_v + j * DV + cb * DN_COLS + c - 2 * DK);
            __half x[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) { const int ri = r1 - 3 + q; x[q] = ri >= r0 ? p.proj[(size_t)ri * p.ld + col] : hist[c * 3 + (ri - r0 + 3)]; }
#pragma unroll
            for (int q = 0; q < 3; ++q) hist[c * 3 + q] = x[q];
        }
        return;
    }
    const int item = blockIdx.x * (DN_THREADS / 32) + (tid >> 5), i = item / p.nv, j = item % p.nv;
    if (i >= r1 - r0) return;
    const float* y = tw + ((size_t)j * n_chunks + i / DC_C) * B::FLOATS + B::U0 + (i % DC_C) * DV + lane * PL;
    const __half* zp = p.proj + (size_t)(r0 + i) * p.ld + p.off_z + j * DV + lane * PL;
    float v[PL], ss = 0.f;
#pragma unroll
    for (int e = 0; e < PL; e += 2) { const float2 f = *(const float2*)(y + e); v[e] = f.x; v[e + 1] = f.y; }
#pragma unroll
    for (int e = 0; e < PL; ++e) ss += v[e] * v[e];
    const float inv = rsqrtf(warp_sum(ss) / (float)DV + p.eps);
    __half* o = p.out + (size_t)(r0 + i) * p.ldo + j * DV + lane * PL;
#pragma unroll
    for (int e = 0; e < PL; ++e) o[e] = __float2half(v[e] * inv * __half2float(p.norm_w[lane * PL + e]) * silu_fast(__half2float(zp[e])));
}

template <int DK, int DV>
static int launch_delta_chunk(const DeltaParams* p, const void* ab, int ld_ab, __half* qk_pre, int ld_qk, int n_rows,
                              float* tw, cudaStream_t s) {
    if (qk_pre) {
        dim3 grid((n_rows + QP_ROWS - 1) / QP_ROWS, (2 * p->nk + 7) / 8);
        if (cudaError_t e = launch_pdl(deltanet_qk_prep_kernel<DK>, grid, dim3(256), 0, s, *p, qk_pre, ld_qk, DV / DN_COLS, 2 * DK + DN_COLS)) return e;
    }
    if (qk_pre && tw) {
        const int n_chunks = (n_rows + DC_C - 1) / DC_C;
        constexpr size_t psm = (size_t)(2 * DC_C * DC_LDK(DK) + DC_C * (DV + 8) + 3 * DC_C * DC_LDA + 2 * DC_C) * sizeof(float);
        static SmemOptIn opt_tw, opt_scan[2];
        if (cudaError_t e = opt_tw.ensure(deltanet_tw_prep_kernel<DK, DV>, psm)) return e;
        if (cudaError_t e = launch_pdl(deltanet_tw_prep_kernel<DK, DV>, dim3(n_chunks, p->nv), dim3(DN_THREADS), psm, s, *p, (const __half*)ab, ld_ab, qk_pre, ld_qk, tw, n_chunks)) return e;
        // (more than half of an SM's shared memory keeps a second CTA off)
        const bool one = p->nv * (DV / 32) <= 148, wide = !one && p->nv * (DV / 64) <= 148;
        const size_t half = 120 * 1024, need = wide ? sizeof(ScanSmem<DK, 64>) : sizeof(ScanSmem<DK, 32>), ssm = (one || wide) && need < half ? half : need;
        const auto scan = wide ? deltanet_scan_kernel<DK, DV, 64> : deltanet_scan_kernel<DK, DV, 32>;
        if (cudaError_t e = opt_scan[wide].ensure(scan, ssm)) return e;
        if (cudaError_t e = launch_pdl(scan, dim3(DV / (wide ? 64 : 32), p->nv), dim3(DN_THREADS), ssm, s, *p, (const __half*)qk_pre, ld_qk, tw, n_chunks)) return e;
        const int row_ctas = (int)(((long long)n_rows * p->nv + DN_THREADS / 32 - 1) / (DN_THREADS / 32));
        return launch_pdl(deltanet_scan_out_kernel<DK, DV>, dim3(row_ctas + p->nv * (DV / DN_COLS)), dim3(DN_THREADS), 0, s, *p, tw, n_chunks, row_ctas);
    }
    constexpr int CB = DV / DN_COLS;
    constexpr int NCH = 2 * DK + DN_COLS;
    size_t smem = (size_t)(2 * DC_C * DC_LDK(DK) + DC_C * DC_LDU + 2 * DC_C * DN_COLS + 2 * DC_C * DC_LDA + DN_COLS * DC_LDK(DK) + NCH * 7 +
                           3 * DC_C + 2 * DC_C) * sizeof(float) + (size_t)(DC_C + 3) * NCH * sizeof(__half);
    static SmemOptIn optin;
    {
        cudaError_t e = optin.ensure(deltanet_chunk_kernel<DK, DV>, smem);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CB, p->nv, p->n_seqs);
    cfg.blockDim = dim3(DN_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CB;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, deltanet_chunk_kernel<DK, DV>, *p, (const __half*)ab, ld_ab, (const __half*)qk_pre, ld_qk);
}

// ab: [rows][ld_ab] fp16 with a at column head and b at column nv + head.
// qk_scratch (optional): fp16 [n_rows][ld_qk >= 2 * nk * dk] work buffer; with it, and ONE launched sequence of
// n_rows rows, the q / k convolution and norms run once in a parallel pre-pass instead of inside the scan.
// tw_scratch (optional, needs qk_scratch): b2_deltanet_tw_floats(nv, n_rows) floats; with it the scan runs in three parts,
// of which only the middle one walks over the chunks.
B2_API int b2_deltanet_chunk(const DeltaParams* p, const void* ab, int ld_ab, void* qk_scratch, int ld_qk, int n_rows,
                             void* tw_scratch, int dk, int dv, cudaStream_t s) {
    if (p->nv % p->nk || !ab) return cudaErrorInvalidValue;
    __half* qk = (__half*)qk_scratch;
    if (qk && (p->n_seqs != 1 || n_rows < 1 || ld_qk < 2 * p->nk * dk || (ld_qk & 7) || ((uintptr_t)qk & 15))) qk = nullptr;
    float* tw = (float*)tw_scratch;
    if (tw && (!qk || ((uintptr_t)tw & 15))) tw = nullptr;
    if (dk == 128 && dv == 128) return launch_delta_chunk<128, 128>(p, ab, ld_ab, qk, ld_qk, n_rows, tw, s);
    if (dk == 64 && dv == 64) return launch_delta_chunk<64, 64>(p, ab, ld_ab, qk, ld_qk, n_rows, tw, s);
    return cudaErrorInvalidValue;
}
B2_API long long b2_deltanet_tw_floats(int nv, int n_rows) { return (long long)nv * ((n_rows + DC_C - 1) / DC_C) * ScanBlock<128, 128>::FLOATS; }

__device__ __forceinline__ void ab_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// a / b gate projections of many rows: ab[t][o] = x[t] . w[o] (o < nv: wa, else wb), a handful of outputs over the whole
// width, so neither a GEMM tile nor a dot product per warp fills the GPU: as one dense tcgen05 launch a CTA walked all of K
// alone, with a warp per output on the FMA pipes 24 rows of 2048 took 9.5 us.  A CTA takes 16 rows x 32 outputs and its 8
// warps divide K in steps of 32; they meet in shared memory.  The order of k inside a product is free, so lane t of a row
// quad takes 8 adjacent k of its rows (16 bytes) and these are its fragments of two mma.sync.  Measured: 8.4 us for 512 rows of
// 5120 and 96 outputs (27 before), 4.8 us for 24 rows of 2048.
// Few rows: there are fewer CTAs than SMs, and the 20 steps of a width of 5120, three on their way at a time, were most of
// the time of a launch that nothing runs beside.  AB_SPLIT CTAs, a cluster, share K then, have all their steps (five) on
// their way at once and add up through distributed shared memory: verification of 80 rows of 5120 (48 such launches) 11.51 -> 11.16 ms, decode
// of 24 rows of 2048 2.88 -> 2.85 ms (12 launches).  What bounds it: one trip to memory, the exchange, and the launch.
#define AB_TOK 16
#define AB_OUT 32
#define AB_WARPS 8
#define AB_SPLIT 4
#define AB_ITEMS (2 + AB_OUT / 8)   // 16-byte pieces of a lane and step: two token rows, four output rows
template <int RING, bool SPLIT>
__global__ void __launch_bounds__(AB_WARPS * 32) ab_proj_kernel(const __half* __restrict__ x, int ldx, const __half* __restrict__ wa,
                                                                const __half* __restrict__ wb, int nv, int H,
                                                                __half* __restrict__ ab, int ld_ab, int rows) {
    extern __shared__ uint4 ab_smem[];               // [AB_WARPS][RING][AB_ITEMS][32 lanes]
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    uint4* ring = ab_smem + warp * (RING * AB_ITEMS * 32) + lane;
    const int r0 = blockIdx.x * AB_TOK, o0 = blockIdx.y * AB_OUT;
    const __half* xr[2];
    const __half* wr[AB_OUT / 8];
#pragma unroll
    for (int i = 0; i < 2; ++i) xr[i] = x + (size_t)min(r0 + g + 8 * i, rows - 1) * ldx + 8 * t;
#pragma unroll
    for (int n = 0; n < AB_OUT / 8; ++n) {
        const int o = min(o0 + 8 * n + g, 2 * nv - 1);
        wr[n] = (o < nv ? wa + (size_t)o * H : wb + (size_t)(o - nv) * H) + 8 * t;
    }
    const int all = (H + AB_WARPS * 32 - 1) / (AB_WARPS * 32), per = SPLIT ? (all + AB_SPLIT - 1) / AB_SPLIT : all;
    const int i0 = SPLIT ? (int)blockIdx.z * per : 0, steps = min(all, i0 + per);
    if (SPLIT) {
        // (into L2 only, where whatever wrote them is seen)
        for (int i = i0; i < steps; ++i) {
            const int k0 = (i * AB_WARPS + warp) * 32;
            if (k0 + 8 * t < H)
#pragma unroll
                for (int n = 0; n < AB_OUT / 8; ++n) asm volatile("prefetch.global.L2 [%0];" :: "l"(wr[n] + k0));
        }
    }
    pdl_wait();
    float acc[AB_OUT / 8][4];
#pragma unroll
    for (int n = 0; n < AB_OUT / 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    // a lane copies what it reads back itself (cp.async), RING - 1 steps ahead: no barrier
    auto issue = [&](int i, int slot) {
        const int k0 = (i * AB_WARPS + warp) * 32;
        uint4* d = ring + slot * AB_ITEMS * 32;
        if (k0 + 8 * t < H) {                        // (H is a multiple of 8)
#pragma unroll
            for (int q = 0; q < 2; ++q) cp_async16(d + q * 32, xr[q] + k0);
#pragma unroll
            for (int n = 0; n < AB_OUT / 8; ++n) cp_async16(d + (2 + n) * 32, wr[n] + k0);
        } else {
#pragma unroll
            for (int q = 0; q < AB_ITEMS; ++q) d[q * 32] = make_uint4(0u, 0u, 0u, 0u);
        }
    };
#pragma unroll
    for (int j = 0; j < RING - 1; ++j) {
        if (i0 + j < steps) issue(i0 + j, j);
        cp_async_commit();
    }
    for (int i = i0; i < steps; ++i) {
        if (i + RING - 1 < steps) issue(i + RING - 1, (i - i0 + RING - 1) % RING);
        cp_async_commit();
        cp_async_wait<RING - 1>();
        const uint4* v = ring + ((i - i0) % RING) * AB_ITEMS * 32;
        const uint4 lo = v[0], hi = v[32];
        const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
        for (int n = 0; n < AB_OUT / 8; ++n) {
            const uint4 w = v[(2 + n) * 32];
            float y0[4] = {}, y1[4] = {};        // (from zero: the tensor core cuts its sums off, the additions to acc round)
            ab_mma(y0, a0, w.x, w.y);
            ab_mma(y1, a1, w.z, w.w);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] += y0[e] + y1[e];
        }
    }
    __syncthreads();                                 // the partial sums take the ring's place
    float (*red)[AB_TOK][AB_OUT + 2] = (float (*)[AB_TOK][AB_OUT + 2])ab_smem;
#pragma unroll
    for (int n = 0; n < AB_OUT / 8; ++n) {
        *(float2*)&red[warp][g][8 * n + 2 * t] = make_float2(acc[n][0], acc[n][1]);
        *(float2*)&red[warp][g + 8][8 * n + 2 * t] = make_float2(acc[n][2], acc[n][3]);
    }
    __syncthreads();
    float* part = (float*)(red + AB_WARPS);          // this CTA's share of the sums (SPLIT)
    for (int i = tid; i < AB_TOK * AB_OUT; i += AB_WARPS * 32) {
        const int r = i / AB_OUT, o = i % AB_OUT;
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < AB_WARPS; ++w) s += red[w][r][o];
        if (SPLIT) { part[i] = s; continue; }
        if (r0 + r < rows && o0 + o < 2 * nv) ab[(size_t)(r0 + r) * ld_ab + o0 + o] = __float2half(s);
    }
    if (SPLIT) {
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        constexpr int EACH = AB_TOK * AB_OUT / AB_SPLIT;     // every CTA ends a share of the tile
        if (tid < EACH) {
            const int i = (int)blockIdx.z * EACH + tid, r = i / AB_OUT, o = i % AB_OUT;
            float v[AB_SPLIT], s = 0.f;
#pragma unroll
            for (int z = 0; z < AB_SPLIT; ++z) v[z] = cl.map_shared_rank(part, z)[i];
#pragma unroll
            for (int z = 0; z < AB_SPLIT; ++z) s += v[z];
            if (r0 + r < rows && o0 + o < 2 * nv) ab[(size_t)(r0 + r) * ld_ab + o0 + o] = __float2half(s);
        }
        cl.sync();                                   // (no CTA leaves while its sums are read)
    }
}
B2_API int b2_ab_proj(const void* x, int ldx, const void* wa, const void* wb, int nv, int H, void* ab, int ld_ab,
                      int rows, cudaStream_t s) {
    if (H % 8 || (ldx % 8)) return cudaErrorInvalidValue;
    const dim3 tiles((rows + AB_TOK - 1) / AB_TOK, (2 * nv + AB_OUT - 1) / AB_OUT);
    auto smem = [](int ring) { return (size_t)AB_WARPS * ring * AB_ITEMS * 32 * 16; };
    static SmemOptIn optin[2];
    // with at most 148 CTAs in all, and a step at least for each of them
    if (tiles.x * tiles.y * AB_SPLIT <= 148 && (H + AB_WARPS * 32 - 1) / (AB_WARPS * 32) >= AB_SPLIT) {
        auto kern = ab_proj_kernel<6, true>;
        if (cudaError_t e = optin[0].ensure(kern, smem(6))) return e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(tiles.x, tiles.y, AB_SPLIT); cfg.blockDim = dim3(AB_WARPS * 32); cfg.dynamicSmemBytes = smem(6); cfg.stream = s;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = AB_SPLIT;
        cfg.attrs = attr; cfg.numAttrs = 2;
        return cudaLaunchKernelEx(&cfg, kern, (const __half*)x, ldx, (const __half*)wa, (const __half*)wb, nv, H, (__half*)ab, ld_ab, rows);
    }
    auto kern = ab_proj_kernel<4, false>;
    if (cudaError_t e = optin[1].ensure(kern, smem(4))) return e;
    return launch_pdl(kern, tiles, dim3(AB_WARPS * 32), smem(4), s, (const __half*)x, ldx, (const __half*)wa, (const __half*)wb, nv, H, (__half*)ab, ld_ab, rows);
}
