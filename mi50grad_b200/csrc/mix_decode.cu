// Both halves of a parallel mixer in one launch, for decode: the windowed attention and the recurrence read what
// mix_prepare left and write columns of their own of one output row, so they need not wait for one another.  As two
// launches the second paid its own start and the end of the first: decode of one sequence at width 4096 (64 heads of 128 x 64, context
// 1500, eight layers) 1.187 -> 1.125 ms a token.  What bounds it: the chain of loads, sums and the last CTA's merge in each role.
#include "window_decode.cuh"
#include "ssd_step.cuh"

// CTAs [0, n_attn): attention, (G, rows, splits) with G fastest; then the recurrence, (heads, column blocks, sequences).
// Two on an SM, as the attention alone with at most four query heads of at most 128 a CTA: wider heads keep more registers,
// and then the recurrence would wait for the attention's SMs.
template <typename T, int EPL, int GT, int NB>
__global__ void __launch_bounds__(WD_THREADS, 2) mix_decode_kernel(const MixLayer L, const MixRun R, const int n_attn, const int col_blocks) {
    static_assert(WD_THREADS == SS_THREADS, "one CTA size for both roles");
    pdl_launch_dependents();
    int b = blockIdx.x;
    if (b < n_attn) {
        const int row = b / L.G % R.n_rows;
        window_decode_cta<T, EPL, GT, false>(L, R, b % L.G, row, b / (L.G * R.n_rows));
        return;
    }
    b -= n_attn;
    ssd_step_cta<T, NB, 1>(L, R, b % L.heads, b / L.heads % col_blocks, col_blocks, b / (L.heads * col_blocks));
}

template <typename T, int EPL, int GT>
static int launch_md(const MixLayer* l, const MixRun* run, cudaStream_t s) {
    MixRun r = *run;
    r.splits = window_decode_splits(l, run, 2 * 148);
    const int n_attn = l->G * r.n_rows * r.splits, cb = (l->P + 31) / 32;
    const dim3 grid(n_attn + l->heads * cb * r.n_seqs);
    if (l->N <= 64) return launch_pdl(mix_decode_kernel<T, EPL, GT, 8>, grid, dim3(WD_THREADS), 0, s, *l, r, n_attn, cb);
    return launch_pdl(mix_decode_kernel<T, EPL, GT, 16>, grid, dim3(WD_THREADS), 0, s, *l, r, n_attn, cb);
}
template <typename T, int EPL>
static int launch_md_heads(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    const int Gq = l->H / l->G;
    return Gq <= 1 ? launch_md<T, EPL, 1>(l, r, s) : Gq <= 2 ? launch_md<T, EPL, 2>(l, r, s) : launch_md<T, EPL, 4>(l, r, s);
}
template <typename T>
static int launch_md_t(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    return l->dp <= 64 ? launch_md_heads<T, 2>(l, r, s) : launch_md_heads<T, 4>(l, r, s);
}

// One row a sequence, plain windows, at most four query heads a key head of at most 128, states of at most 128; and all CTAs
// resident at once: beyond that the recurrence, which alone has three CTAs on an SM, is slowed more than a launch costs (seven
// sequences of 64 heads, 960 CTAs: decode of 7 tokens 11.37 ms merged, 11.27 apart).
B2_API int b2_mix_decode_takes(const MixLayer* l, const MixRun* r) {
    return attn_valid(l) && ssd_valid(l) && r->n_seqs >= 1 && r->n_rows == r->n_seqs && r->fuse_norm && r->splits >= 1 && r->splits <= WD_MAX_SPLITS &&
           l->keep_first <= 0 && l->softcap <= 0.f && !l->sink && l->dv == l->d && l->vp == l->dp && l->H / l->G <= 4 && l->dp <= 128 && l->N <= 128 &&
           l->G * r->n_rows * window_decode_splits(l, r, 2 * 148) + l->heads * ((l->P + 31) / 32) * r->n_seqs <= 2 * 148;
}
B2_API int b2_mix_decode(const MixLayer* l, const MixRun* r, cudaStream_t s) {
    if (!b2_mix_decode_takes(l, r)) return cudaErrorInvalidValue;
    return r->dt == DT_BF16 ? launch_md_t<bf16>(l, r, s) : launch_md_t<float>(l, r, s);
}
