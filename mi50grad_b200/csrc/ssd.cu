// Linear recurrences with a scalar decay per head and token:
//     S_t = a_t S_(t-1) + dt_t B_t x_t^T,     y_t = S_t^T C_t + D x_t
// with S [N x P] fp32 per head, B and C shared by the heads of a group.
//   Mamba-2 (state-space duality): a_t = exp(-exp(A_log) dt_t); then an RMSNorm of y * silu(z) in ngroups parts.
//   Lightning attention: a constant per head, dt = 1, no D, q / k / v in the places of C / B / x, every head its own
//   group; then an RMSNorm of y times sigmoid(z).
//
//   ssd_step    token by token: one CTA per (head, 32 columns of P, sequence), the state in registers
//               (requested before the dependency wait); the last CTA of a norm part normalises it.
//   ssd_chunk   prompts in bf16: chunks of 64 tokens.  (1) local end state of every chunk, (2) the pass over
//               the chunks, (3) outputs.  The products run on bf16 tensor cores; every operand that is not
//               exactly bf16 (weighted inputs, masked scores, states) enters as the sum of three bf16 terms
//               (24 bits), so the recurrence keeps fp32 accuracy.
#include "mixers.cuh"
#include "ssd_step.cuh"

template <typename T>
__global__ void __launch_bounds__(256) ssd_norm_kernel(const MixLayer L, const MixRun R) {
    __shared__ float red[32];
    pdl_launch_dependents();
    pdl_wait();
    norm_part<T>(L, R, blockIdx.x, blockIdx.y, red);
}

// ---------------------------------------------------------------------------
// token by token: grid (heads, ceil(P / 32), sequences); lane = column of P, warp = slice of N
// ---------------------------------------------------------------------------
template <typename T, int NB, int U>
__global__ void __launch_bounds__(SS_THREADS) ssd_step_kernel(const MixLayer L, const MixRun R) {
    pdl_launch_dependents();
    ssd_step_cta<T, NB, U>(L, R, blockIdx.x, blockIdx.y, gridDim.y, blockIdx.z);
}

// one CTA per part of a row, with a thread for every four columns of it
template <typename T>
static int launch_ssd_norm(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    const int w4 = (l->heads * l->P / l->ngroups + 3) / 4, nt = w4 >= 256 ? 256 : (w4 + 31) / 32 * 32;
    return launch_pdl(ssd_norm_kernel<T>, dim3(r->n_rows, l->ngroups), dim3(nt), 0, s, *l, *r);
}
template <typename T>
static int launch_ssd_step(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    dim3 grid(l->heads, (l->P + 31) / 32, r->n_seqs);
    // one token a sequence, as in decode, has nothing to overlap
    auto go = [&](auto one, auto many) { return launch_pdl(r->n_rows > r->n_seqs ? many : one, grid, dim3(SS_THREADS), 0, s, *l, *r); };
    int e;
    if (l->N <= 64) e = go(ssd_step_kernel<T, 8, 1>, ssd_step_kernel<T, 8, 8>);
    else if (l->N <= 128) e = go(ssd_step_kernel<T, 16, 1>, ssd_step_kernel<T, 16, 8>);
    else e = go(ssd_step_kernel<T, 32, 1>, ssd_step_kernel<T, 32, 4>);
    if (e || r->fuse_norm) return e;
    return launch_ssd_norm<T>(l, r, s);
}
// Any mix of sequences; fuse_norm = 0 adds a launch for the norm (many rows per sequence).
B2_API int b2_ssd_step(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    if (!ssd_valid(l) || r->n_seqs < 1) return cudaErrorInvalidValue;
    return r->dt == DT_BF16 ? launch_ssd_step<bf16>(l, r, s) : launch_ssd_step<float>(l, r, s);
}
B2_API int b2_ssd_units(const MixLayer* l, int n_seqs) { return n_seqs * (l->heads % l->ngroups ? 1 : l->ngroups); }

// ---------------------------------------------------------------------------
// chunked scan: one sequence, bf16
// ---------------------------------------------------------------------------
#define SC_T SSD_CHUNK
#define SC_P 64                  // columns of P per CTA
#define SC_LDP (SC_P + 8)
#define SC_TERMS 3

__device__ __forceinline__ void sc_ldsm4(uint32_t (&r)[4], const bf16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void sc_ldsm4_t(uint32_t (&r)[4], const bf16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void sc_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// v = t[0] + t[1] + t[2] with bf16 terms (exact to 24 bits)
__device__ __forceinline__ void sc_split(float v, bf16 (&t)[SC_TERMS]) {
#pragma unroll
    for (int i = 0; i < SC_TERMS; ++i) { t[i] = __float2bfloat16(v); v -= __bfloat162float(t[i]); }
}

// cumulative log decay of a chunk (one warp; two tokens per lane)
__device__ __forceinline__ void sc_cumsum(const MixLayer& L, const MixRun& R, int t0, int n, int h, float A, float* la, float* dts, int lane) {
    const float d0 = 2 * lane < n ? rec_dt(L, R, t0 + 2 * lane, h) : 0.f;
    const float d1 = 2 * lane + 1 < n ? rec_dt(L, R, t0 + 2 * lane + 1, h) : 0.f;
    const float a0 = A * d0, a1 = A * d1;
    float s = a0 + a1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const float v = __shfl_up_sync(0xffffffffu, s, o); if (lane >= o) s += v; }
    const float before = s - (a0 + a1);
    la[2 * lane] = before + a0; la[2 * lane + 1] = s;
    dts[2 * lane] = d0; dts[2 * lane + 1] = d1;
}
// rows [t0, t0 + n) x columns [c0, c0 + w) of xbc into smem [64][ld], zero-padded to wp columns (wp % 8 == 0)
__device__ __forceinline__ void sc_stage(const MixRun& R, int t0, int n, int c0, int w, int wp, bf16* dst, int ld, int tid, int nthr) {
    const bf16* src = (const bf16*)R.xbc + c0;
    const bool vec = ((R.ld_xbc | c0) & 7) == 0 && ((uintptr_t)R.xbc & 15) == 0;
    const int ppr = wp >> 3, sh = ppr > 1 ? 32 - __clz(ppr - 1) : 0, c = (tid & ((1 << sh) - 1)) * 8;      // (no division for each piece)
    if (c < wp)
        for (int r = tid >> sh; r < SC_T; r += nthr >> sh) {
            bf16* d = dst + r * ld + c;
            if (vec && r < n && c + 8 <= w) cp_async16(d, src + (size_t)(t0 + r) * R.ld_xbc + c);
            else
#pragma unroll
                for (int e = 0; e < 8; ++e) d[e] = (r < n && c + e < w) ? src[(size_t)(t0 + r) * R.ld_xbc + c + e] : __float2bfloat16(0.f);
        }
    cp_async_commit();
}

// (1) local end states: grid (chunks, heads, ceil(P / 64)), four warps over the rows of N
__global__ void __launch_bounds__(128) ssd_chunk_state_kernel(const MixLayer L, const MixRun R) {
    extern __shared__ __align__(16) unsigned char sc_smem[];
    const int Np = (L.N + 15) & ~15, LDN = Np + 8;
    bf16* Bs = (bf16*)sc_smem;                               // [64][LDN]
    bf16* W = Bs + SC_T * LDN;                               // [3][64][SC_LDP]
    __shared__ float la[SC_T], dts[SC_T];
    pdl_launch_dependents();
    const int c = blockIdx.x, h = blockIdx.y, p0 = blockIdx.z * SC_P;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int grp = h / (L.heads / L.groups), pw = min(SC_P, L.P - p0);
    const int t0 = c * SC_T, n = min(SC_T, R.n_rows - t0);
    const float A = rec_rate(L, h);
    pdl_wait();
    sc_stage(R, t0, n, L.rB + grp * L.N, L.N, Np, Bs, LDN, tid, 128);
    // x in pieces of eight columns, all of a thread's requested at once: element by element between the stores of W they were
    // a trip to L2 each (1000 rows, 80 heads of 128 x 64: 63 -> 29 us, bound by its shared-memory traffic now)
    constexpr int PIECES = SC_T * (SC_P / 8) / 128;
    uint4 xr[PIECES];
    const int x0 = L.rx + h * L.P + p0;
    const bool vec = ((R.ld_xbc | x0) & 7) == 0 && ((uintptr_t)R.xbc & 15) == 0;
#pragma unroll
    for (int j = 0; j < PIECES; ++j) {
        const int i = tid + 128 * j, s = i / (SC_P / 8), p = i % (SC_P / 8) * 8;
        const bf16* src = (const bf16*)R.xbc + (size_t)(t0 + s) * R.ld_xbc + x0 + p;
        if (s < n && vec && p + 8 <= pw) xr[j] = *(const uint4*)src;
        else {
            bf16 e8[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) e8[e] = s < n && p + e < pw ? src[e] : __float2bfloat16(0.f);
            xr[j] = make_uint4(sc_pack(e8[0], e8[1]), sc_pack(e8[2], e8[3]), sc_pack(e8[4], e8[5]), sc_pack(e8[6], e8[7]));
        }
    }
    if (warp == 0) sc_cumsum(L, R, t0, n, h, A, la, dts, lane);
    __syncthreads();
    const float end = la[SC_T - 1];
#pragma unroll
    for (int j = 0; j < PIECES; ++j) {
        const int i = tid + 128 * j, s = i / (SC_P / 8), p = i % (SC_P / 8) * 8;
        const float f = s < n ? dts[s] * expf(end - la[s]) : 0.f;
        const uint32_t w[4] = {xr[j].x, xr[j].y, xr[j].z, xr[j].w};
        uint32_t o[SC_TERMS][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            bf16 q0[SC_TERMS], q1[SC_TERMS];
            sc_split(__uint_as_float(w[e] << 16) * f, q0);
            sc_split(__uint_as_float(w[e] & 0xffff0000u) * f, q1);
#pragma unroll
            for (int k = 0; k < SC_TERMS; ++k) o[k][e] = sc_pack(q0[k], q1[k]);
        }
#pragma unroll
        for (int k = 0; k < SC_TERMS; ++k) *(uint4*)(W + (k * SC_T + s) * SC_LDP + p) = make_uint4(o[k][0], o[k][1], o[k][2], o[k][3]);
    }
    cp_async_wait<0>();
    __syncthreads();
    const int g = lane >> 2, t = lane & 3;
    const int v_row = (lane & 7) + ((lane >> 3) & 1) * 8, v_col = (lane >> 4) * 8;
    float* out = R.chunk_state + ((size_t)c * L.heads + h) * L.N * L.P + p0;
    const bool pairs = (L.P & 1) == 0 && ((uintptr_t)R.chunk_state & 7) == 0;
    for (int mt = warp; mt < Np / 16; mt += 4) {
        float acc[SC_P / 8][4];
#pragma unroll
        for (int j = 0; j < SC_P / 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
#pragma unroll
        for (int k0 = 0; k0 < SC_T; k0 += 16) {
            uint32_t a[4];                                   // A = B^T: (m = state row, k = token) from [token][state row]
            sc_ldsm4_t(a, Bs + (k0 + (lane & 7) + (lane >> 4) * 8) * LDN + mt * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
            for (int q = 0; q < SC_TERMS; ++q)
#pragma unroll
                for (int np = 0; np < SC_P / 16; ++np) {
                    if (np * 16 >= pw) break;
                    uint32_t b[4];
                    sc_ldsm4_t(b, W + (q * SC_T + k0 + v_row) * SC_LDP + np * 16 + v_col);
                    sc_mma(acc[2 * np], a, b[0], b[1]);
                    sc_mma(acc[2 * np + 1], a, b[2], b[3]);
                }
        }
#pragma unroll
        for (int j = 0; j < SC_P / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
                const int nn = mt * 16 + g + 4 * e, p = 8 * j + 2 * t;
                if (nn >= L.N || p >= pw) continue;
                float* o = out + (size_t)nn * L.P + p;
                if (pairs) *(float2*)o = make_float2(acc[j][e], acc[j][e + 1]);
                else { o[0] = acc[j][e]; if (p + 1 < pw) o[1] = acc[j][e + 1]; }
            }
    }
    if (tid == 0 && blockIdx.z == 0) R.chunk_decay[c * L.heads + h] = end;
    // nothing of this launch reads the convolution history: carry it over here
    if (c == 0 && R.commit) conv_history_of<bf16>(L, R, R.rows[0].seq, 0, R.n_rows, h, p0, SC_P, tid, 128);
}

#define SC_AHEAD 4               // chunks whose states are requested at once

// (2) the pass over the chunks: grid (ceil(N * Pp / 256), heads); leaves the state before every chunk as bf16 planes
__global__ void __launch_bounds__(256) ssd_chunk_pass_kernel(const MixLayer L, const MixRun R, int chunks) {
    pdl_launch_dependents();
    if (!R.older) pdl_wait();
    const int Pp = (L.P + 7) & ~7, h = blockIdx.y;
    const int i = blockIdx.x * 256 + threadIdx.x, n = i / Pp, p = i % Pp;
    const bool in = n < L.N, ok = in && p < L.P;
    float* S = L.state + (((size_t)R.rows[0].seq * L.heads + h) * L.N + n) * L.P + p;
    float s = ok ? *S : 0.f;
    pdl_wait();
    if (!in) return;
    const float* cs = R.chunk_state + ((size_t)h * L.N + n) * L.P + p;
    const size_t cst = (size_t)L.heads * L.N * L.P;
    bf16* prev = (bf16*)R.chunk_prev + ((size_t)h * SC_TERMS * L.N + n) * Pp + p;
    const size_t pst = (size_t)L.heads * SC_TERMS * L.N * Pp;
    for (int c0 = 0; c0 < chunks; c0 += SC_AHEAD) {
        float v[SC_AHEAD], d[SC_AHEAD];
#pragma unroll
        for (int u = 0; u < SC_AHEAD; ++u) {
            v[u] = (ok && c0 + u < chunks) ? cs[(c0 + u) * cst] : 0.f;
            d[u] = c0 + u < chunks ? R.chunk_decay[(c0 + u) * L.heads + h] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < SC_AHEAD; ++u) {
            if (c0 + u >= chunks) break;
            bf16 q[SC_TERMS];
            sc_split(s, q);
#pragma unroll
            for (int k = 0; k < SC_TERMS; ++k) prev[(c0 + u) * pst + (size_t)k * L.N * Pp] = q[k];
            s = fmaf(expf(d[u]), s, v[u]);
        }
    }
    if (ok && R.commit) *S = s;
}

// (3) outputs: grid (chunks, heads, ceil(P / 64)), four warps of 16 tokens
__global__ void __launch_bounds__(128) ssd_chunk_out_kernel(const MixLayer L, const MixRun R) {
    extern __shared__ __align__(16) unsigned char sc_smem[];
    const int Np = (L.N + 15) & ~15, LDN = Np + 8, Pp = (L.P + 7) & ~7;
    bf16* Cs = (bf16*)sc_smem;                               // [64][LDN]
    bf16* Bs = Cs + SC_T * LDN;                              // [64][LDN]
    bf16* Xs = Bs + SC_T * LDN;                              // [64][SC_LDP]
    bf16* Sp = Xs + SC_T * SC_LDP;                           // [3][Np][SC_LDP]
    __shared__ float la[SC_T], dts[SC_T];
    pdl_launch_dependents();
    const int c = blockIdx.x, h = blockIdx.y, p0 = blockIdx.z * SC_P;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int grp = h / (L.heads / L.groups), pw = min(SC_P, L.P - p0), pwp = (pw + 7) & ~7;
    const int t0 = c * SC_T, n = min(SC_T, R.n_rows - t0);
    const float A = rec_rate(L, h), Dh = L.D ? L.D[h] : 0.f;
    const bool gated = L.gate == REC_GATE_SILU_NORM;
    pdl_wait();
    sc_stage(R, t0, n, L.rC + grp * L.N, L.N, Np, Cs, LDN, tid, 128);
    sc_stage(R, t0, n, L.rB + grp * L.N, L.N, Np, Bs, LDN, tid, 128);
    sc_stage(R, t0, n, L.rx + h * L.P + p0, pw, SC_P, Xs, SC_LDP, tid, 128);
    {
        const bf16* src = (const bf16*)R.chunk_prev + ((size_t)c * L.heads + h) * SC_TERMS * L.N * Pp + p0;
        const int col = tid % (SC_P / 8) * 8;
        for (int nn = tid / (SC_P / 8); nn < Np; nn += 128 / (SC_P / 8))
#pragma unroll
            for (int q = 0; q < SC_TERMS; ++q) {
                bf16* d = Sp + (q * Np + nn) * SC_LDP + col;
                if (nn < L.N && col < pwp) cp_async16(d, src + ((size_t)q * L.N + nn) * Pp + col);
                else *(uint4*)d = make_uint4(0u, 0u, 0u, 0u);
            }
        cp_async_commit();
    }
    // The gates of this lane's outputs are requested here: read between the stores of the outputs, they were a trip to L2
    // for each of 32 elements (1000 rows, 80 heads of 128 x 64: 124 -> 84 us, with staging free of divisions; bound by the instructions of eight
    // warps an SM, a third of them the splits into three terms)
    const int zc = L.off_z + h * L.P + p0;
    const bool z2 = ((zc | R.ld_proj) & 1) == 0 && ((uintptr_t)R.proj & 3) == 0;
    uint32_t zz[SC_P / 8][2];
#pragma unroll
    for (int j = 0; j < SC_P / 8; ++j)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int r = warp * 16 + g + 8 * hf, p = 8 * j + 2 * t;
            const bf16* z = (const bf16*)R.proj + (size_t)(t0 + r) * R.ld_proj + zc + p;
            zz[j][hf] = 0u;
            if (!gated || r >= n || p >= pw) continue;
            if (z2 && p + 1 < pw) zz[j][hf] = *(const uint32_t*)z;
            else zz[j][hf] = sc_pack(z[0], p + 1 < pw ? z[1] : __float2bfloat16(0.f));
        }
    if (warp == 0) sc_cumsum(L, R, t0, n, h, A, la, dts, lane);
    cp_async_wait<0>();
    __syncthreads();
    if (warp * 16 >= n) return;
    const int a_row = (lane & 7) + ((lane >> 3) & 1) * 8, a_col = (lane >> 4) * 8;
    const int b_row = (lane & 7) + (lane >> 4) * 8, b_col = ((lane >> 3) & 1) * 8;
    const bf16* Cw = Cs + warp * 16 * LDN;
    float o[SC_P / 8][4], s[SC_T / 8][4];
#pragma unroll
    for (int j = 0; j < SC_P / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
#pragma unroll
    for (int j = 0; j < SC_T / 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
    for (int k0 = 0; k0 < Np; k0 += 16) {
        uint32_t a[4];
        sc_ldsm4(a, Cw + a_row * LDN + k0 + a_col);
        // scores C B^T of the tokens up to this warp's own
#pragma unroll
        for (int np = 0; np < SC_T / 16; ++np) {
            if (np > warp) break;
            uint32_t b[4];
            sc_ldsm4(b, Bs + (np * 16 + b_row) * LDN + k0 + b_col);
            sc_mma(s[2 * np], a, b[0], b[1]);
            sc_mma(s[2 * np + 1], a, b[2], b[3]);
        }
        // C times the state before the chunk
#pragma unroll
        for (int q = 0; q < SC_TERMS; ++q)
#pragma unroll
            for (int np = 0; np < SC_P / 16; ++np) {
                if (np * 16 >= pw) break;
                uint32_t b[4];
                sc_ldsm4_t(b, Sp + (q * Np + k0 + a_row) * SC_LDP + np * 16 + a_col);
                sc_mma(o[2 * np], a, b[0], b[1]);
                sc_mma(o[2 * np + 1], a, b[2], b[3]);
            }
    }
    const int r_lo = warp * 16 + g, r_hi = r_lo + 8;
    const float la_lo = la[r_lo], la_hi = la[r_hi], e_lo = expf(la_lo), e_hi = expf(la_hi);
#pragma unroll
    for (int j = 0; j < SC_P / 8; ++j) { o[j][0] *= e_lo; o[j][1] *= e_lo; o[j][2] *= e_hi; o[j][3] *= e_hi; }
#pragma unroll
    for (int k16 = 0; k16 < SC_T / 16; ++k16) {
        if (k16 > warp) break;
        uint32_t pa[SC_TERMS][4];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int j = 2 * k16 + hf, s0 = 8 * j + 2 * t;
            bf16 q0[SC_TERMS], q1[SC_TERMS], q2[SC_TERMS], q3[SC_TERMS];
            sc_split(s0 <= r_lo ? s[j][0] * expf(la_lo - la[s0]) * dts[s0] : 0.f, q0);
            sc_split(s0 + 1 <= r_lo ? s[j][1] * expf(la_lo - la[s0 + 1]) * dts[s0 + 1] : 0.f, q1);
            sc_split(s0 <= r_hi ? s[j][2] * expf(la_hi - la[s0]) * dts[s0] : 0.f, q2);
            sc_split(s0 + 1 <= r_hi ? s[j][3] * expf(la_hi - la[s0 + 1]) * dts[s0 + 1] : 0.f, q3);
#pragma unroll
            for (int q = 0; q < SC_TERMS; ++q) { pa[q][hf * 2] = sc_pack(q0[q], q1[q]); pa[q][hf * 2 + 1] = sc_pack(q2[q], q3[q]); }
        }
#pragma unroll
        for (int np = 0; np < SC_P / 16; ++np) {
            if (np * 16 >= pw) break;
            uint32_t b[4];
            sc_ldsm4_t(b, Xs + (k16 * 16 + a_row) * SC_LDP + np * 16 + a_col);
#pragma unroll
            for (int q = 0; q < SC_TERMS; ++q) {
                sc_mma(o[2 * np], pa[q], b[0], b[1]);
                sc_mma(o[2 * np + 1], pa[q], b[2], b[3]);
            }
        }
    }
    const bool u2 = ((R.ld_u | (h * L.P + p0)) & 1) == 0 && ((uintptr_t)R.ubuf & 7) == 0;
#pragma unroll
    for (int j = 0; j < SC_P / 8; ++j)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int r = hf ? r_hi : r_lo, p = 8 * j + 2 * t;
            if (r >= n || p >= pw) continue;
            const uint32_t xw = *(const uint32_t*)(Xs + r * SC_LDP + p);
            float u0 = o[j][2 * hf] + Dh * __uint_as_float(xw << 16), u1 = o[j][2 * hf + 1] + Dh * __uint_as_float(xw & 0xffff0000u);
            if (gated) { u0 *= silu_p(__uint_as_float(zz[j][hf] << 16)); u1 *= silu_p(__uint_as_float(zz[j][hf] & 0xffff0000u)); }
            float* u = R.ubuf + (size_t)(t0 + r) * R.ld_u + h * L.P + p0 + p;
            if (u2 && p + 1 < pw) *(float2*)u = make_float2(u0, u1);
            else { u[0] = u0; if (p + 1 < pw) u[1] = u1; }
        }
}

// All rows belong to one sequence, bf16 only (b2_ssd_step takes everything else).
B2_API int b2_ssd_chunk(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    if (!ssd_valid(l) || r->dt != DT_BF16 || r->n_seqs != 1 || !r->chunk_state || !r->chunk_prev || !r->chunk_decay)
        return cudaErrorInvalidValue;
    const int chunks = (r->n_rows + SC_T - 1) / SC_T, Np = (l->N + 15) & ~15, Pp = (l->P + 7) & ~7, pb = (l->P + SC_P - 1) / SC_P;
    const size_t sm1 = ((size_t)SC_T * (Np + 8) + SC_TERMS * SC_T * SC_LDP) * sizeof(bf16);
    const size_t sm3 = ((size_t)2 * SC_T * (Np + 8) + SC_T * SC_LDP + (size_t)SC_TERMS * Np * SC_LDP) * sizeof(bf16);
    static SmemOptIn o1, o3;
    if (int e = o1.ensure((const void*)ssd_chunk_state_kernel, sm1)) return e;
    if (int e = o3.ensure((const void*)ssd_chunk_out_kernel, sm3)) return e;
    if (int e = launch_pdl(ssd_chunk_state_kernel, dim3(chunks, l->heads, pb), dim3(128), sm1, s, *l, *r)) return e;
    if (int e = launch_pdl(ssd_chunk_pass_kernel, dim3((l->N * Pp + 255) / 256, l->heads), dim3(256), 0, s, *l, *r, chunks)) return e;
    if (int e = launch_pdl(ssd_chunk_out_kernel, dim3(chunks, l->heads, pb), dim3(128), sm3, s, *l, *r)) return e;
    return launch_ssd_norm<bf16>(l, r, s);
}
B2_API long long b2_ssd_chunk_state_floats(const MixLayer* l, int rows) {
    return (long long)((rows + SC_T - 1) / SC_T) * l->heads * l->N * l->P;
}
B2_API long long b2_ssd_chunk_prev_bytes(const MixLayer* l, int rows) {
    return (long long)((rows + SC_T - 1) / SC_T) * l->heads * SC_TERMS * l->N * ((l->P + 7) & ~7) * (long long)sizeof(bf16);
}
