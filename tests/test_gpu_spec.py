"""Speculative verification on the device against the fp32 oracle: tree verify, greedy
acceptance, exact commit of DeltaNet state / conv history / KV cache, many-row (tensor-core)
path, and batched decode of more sequences than the GEMV kernels take rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mk(max_batch, seed=0, max_seq=256):
    from mi50grad_b200.config import tiny_config
    from mi50grad_b200.engine.engine import InferenceEngine
    from mi50grad_b200.models.oracle import OracleEngine
    from mi50grad_b200.models.weights import random_model
    cfg = tiny_config()
    mw = random_model(cfg, seed)
    eng = InferenceEngine(cfg, max_seq_len=max_seq, max_batch=max_batch)
    eng.load_model(mw)
    return cfg, mw, eng, OracleEngine(mw, max_seq_len=max_seq, max_batch=max_batch)


def _prompt(cfg, n, seed):
    return torch.randint(0, cfg.vocab_size, (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def _wrong(cfg, *avoid):
    t = 7
    while t in avoid:
        t += 1
    return t % cfg.vocab_size


def test_tree_verify_accepts_oracle_path_and_commits_exactly():
    cfg, mw, eng, orc = _mk(2)
    ids = _prompt(cfg, 12, 1)
    ref, _ = orc.greedy_generate(ids, 9)                  # ref[0] is the pending token after the prompt
    root = eng.prefill_tokens(ids)
    assert root == ref[0]
    g1, g2, g3 = ref[1], ref[2], ref[3]
    # node (draft index): 0 wrong, 1 g1 | below g1: 2 g2, 3 wrong | below g2: 4 wrong
    drafts = [_wrong(cfg, g1), g1, g2, _wrong(cfg, g2), _wrong(cfg, g3)]
    parents = [-1, -1, 1, 1, 2]
    (acc, nxt), = eng.spec_step([drafts], [parents], [0])
    assert acc == [g1, g2] and nxt == g3
    assert eng.states.length(0) == 12 + 3 and eng.states.token(0) == g3
    # the state must be what feeding root, g1, g2 one at a time leaves
    cfg2, _, eng2, _ = _mk(2)
    eng2.prefill_tokens(ids)
    eng2.decode_tokens(3, graph=False)
    S1, S2 = eng.states.dn.S[:, 0], eng2.states.dn.S[:, 0]
    assert (S1 - S2).abs().max() <= 2e-3 * max(1.0, S2.abs().max().item())
    assert torch.equal(eng.states.dn.conv[:, 0], eng2.states.dn.conv[:, 0])
    n = 15
    k1, k2 = eng.states.kv.k[:, 0, :n].float(), eng2.states.kv.k[:, 0, :n].float()
    assert (k1 - k2).abs().max() <= 2e-2 * max(1.0, k2.abs().max().item())
    # and decoding continues like the oracle
    cont = eng.decode_tokens(5, graph=False)[:, 0].tolist()
    assert [g3] + cont == ref[3:9]


def test_chain_speculation_through_generator_equals_greedy():
    from mi50grad_b200.generate.sampler import SamplingParams
    from mi50grad_b200.generate.speculative import SpeculativeGenerator
    from mi50grad_b200.generate.tree_speculative import TreeSpeculativeDecoder
    cfg, mw, eng, orc = _mk(1, seed=3)
    ids = ([11, 22, 33, 44, 55] * 4)[:18]
    ref, _ = orc.greedy_generate(ids, 20)
    gen = SpeculativeGenerator(eng, ngram_size=3, max_draft_len=4)
    out = gen.generate_ids(ids, SamplingParams(temperature=0.0, max_tokens=20))
    assert out == ref
    assert gen.last_stats["forward_passes"] == gen.last_stats["iterations"] + 1   # one pass per iteration + prefill
    dec = TreeSpeculativeDecoder(eng, max_tree_size=6, max_depth=3, branching_factor=2)
    assert dec.generate_ids(ids, 14) == ref[:14]


def test_many_row_verify_three_sequences_tensor_core_path():
    cfg, mw, eng, orc = _mk(4, seed=5)
    prompts = [_prompt(cfg, 17, 10), _prompt(cfg, 9, 11), _prompt(cfg, 20, 12)]
    refs = [orc.greedy_generate(p, 8, seq=i)[0] for i, p in enumerate(prompts)]
    for i, p in enumerate(prompts):
        assert eng.prefill_tokens(p, seq=i) == refs[i][0]
    drafts, parents, expect = [], [], []
    for i, r in enumerate(refs):
        n_ok = i                                           # sequence i accepts i drafts of a 3-chain
        d = [r[1 + k] if k < n_ok else _wrong(cfg, r[1 + k]) for k in range(3)]
        drafts.append(d)
        parents.append([-1, 0, 1])
        expect.append((d[:n_ok], r[1 + n_ok]))
    res = eng.spec_step(drafts, parents, [0, 1, 2])        # 12 rows: beyond the GEMV kernels' 8
    assert [(a, n) for a, n in res] == expect
    assert eng.states.lengths()[:3] == [17 + 1, 9 + 2, 20 + 3]
    out = eng.decode_tokens(3, seqs=[0, 1, 2], graph=False).cpu()
    for i, r in enumerate(refs):
        n_ok = i
        assert [r[1 + n_ok]] + out[:, i].tolist()[:2] == r[1 + n_ok:4 + n_ok][:3]


def test_batched_decode_more_sequences_than_gemv_rows():
    cfg, mw, eng, orc = _mk(10, seed=6, max_seq=64)
    prompts = [_prompt(cfg, 5 + i, 20 + i) for i in range(10)]
    refs = [orc.greedy_generate(p, 4, seq=i)[0] for i, p in enumerate(prompts)]
    for i, p in enumerate(prompts):
        assert eng.prefill_tokens(p, seq=i) == refs[i][0]
    out_e = eng.decode_tokens(3, seqs=list(range(10)), graph=False).cpu()
    for i in range(10):
        assert out_e[:, i].tolist() == refs[i][1:4], i
    assert eng.states.lengths() == [5 + i + 3 for i in range(10)]
    # the same step replayed from a captured graph
    out_g = eng.decode_tokens(2, seqs=list(range(10)), graph=True).cpu()
    assert out_g.shape == (2, 10)


def test_tp_engine_tree_hooks_match_oracle():
    from helpers import cosine
    from mi50grad_b200.config import tiny_config
    from mi50grad_b200.engine.tp_engine import TPInferenceEngine
    from mi50grad_b200.generate.tree_attention import TreeAttentionMask, TreeTopology
    from mi50grad_b200.models.oracle import OracleEngine
    from mi50grad_b200.models.weights import random_model
    cfg = tiny_config()
    mw = random_model(cfg, 4)
    eng = TPInferenceEngine(cfg, max_seq_len=128)
    eng.load_model(mw)
    orc = OracleEngine(mw, max_seq_len=128)
    ids = _prompt(cfg, 10, 31)
    eng.prefill_tokens(ids)
    orc.forward(orc.embed(ids))
    toks, parents = [5, 6, 7, 8, 9, 10], [-1, 0, 0, 1, 1, 2]
    topo = TreeTopology.from_parents(toks, parents)
    embs = orc.embed(toks)
    ref = orc.final_norm(orc.forward(embs, parents=parents))
    S_before = eng.engine.states.dn.S.clone()
    hs = eng.decode_step_tree([e.numpy() for e in embs], TreeAttentionMask(topo, kv_len=10))
    assert torch.equal(S_before, eng.engine.states.dn.S) and eng.engine.states.length(0) == 10
    for i in range(len(toks)):
        assert cosine(torch.from_numpy(hs[i]).float(), ref[i]) > 0.999, i
    hs2, n = eng.decode_step_speculative([e for e in embs[:3]], 10, [6, 7])
    ref2 = orc.final_norm(orc.forward(embs[:3], parents=[-1, 0, 1]))
    assert n == 2 and all(cosine(hs2[i].float().cpu(), ref2[i]) > 0.999 for i in range(3))
    eng.set_eagle_mode(True, k_draft=3)
    d = eng.generate_eagle_drafts(hs[0], 3)
    assert len(d) == 3 and d[0] == int(torch.argmax(orc.compute_logits(ref[0])))


def _tree(n, kind):
    if kind == "chain":
        return [i - 1 for i in range(n)]
    g = torch.Generator().manual_seed(n)
    return [-1] + [int(torch.randint(-1 if kind == "forest" else 0, i, (1,), generator=g)) for i in range(1, n)]


@pytest.mark.parametrize("dk,nk,nv,sizes,kind,ab", [(128, 2, 6, [5, 1, 16], "chain", "proj"), (128, 1, 2, [16, 4, 7], "tree", "lazy"),
                                                    (64, 2, 4, [3, 16, 9], "forest", "proj"), (64, 1, 1, [8], "tree", "xn")])
def test_verify_outputs_equal_steps_along_every_path(dk, nk, nv, sizes, kind, ab):
    """The output of every node of a draft tree is that of feeding its path to the step kernel, token by token; both
    are fp32 sums rounded to fp16 once, so they differ by an ulp or so."""
    import ctypes as C
    from mi50grad_b200.ops import kernels as K
    from mi50grad_b200.ops import lib as L
    g = torch.Generator().manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    dv, H, R, ns = dk, 512, sum(sizes), len(sizes)
    kd = nk * dk
    conv_dim = 2 * kd + nv * dv
    ld = conv_dim + nv * dv + 2 * nv
    proj = rnd(R, ld).half().cuda()
    conv_w, A_log = (rnd(conv_dim, 4) * 0.3).half().cuda(), (torch.rand(nv, generator=g) * 1.5 - 1.0).cuda()
    dt_bias, norm_w = (rnd(nv) * 0.5).half().cuda(), (torch.rand(dv, generator=g) + 0.5).half().cuda()
    state, hist0 = (rnd(ns, nv, dk, dv) * 0.1).cuda(), rnd(ns, conv_dim, 3).half()
    conv = torch.zeros(ns, nv, dv // 32, 2 * dk + 32, 3, dtype=torch.float16)
    for j in range(nv):
        kh = j // (nv // nk)
        for cb in range(dv // 32):
            ch = [kh * dk + i for i in range(dk)] + [kd + kh * dk + i for i in range(dk)] + [2 * kd + j * dv + cb * 32 + i for i in range(32)]
            conv[:, j, cb] = hist0[:, ch]
    conv = conv.cuda()
    wa, wb, xn = (rnd(nv, H) * 0.05).half().cuda(), (rnd(nv, H) * 0.05).half().cuda(), rnd(R, H).half().cuda()
    hres, wnorm = (rnd(R, H) * 3).cuda(), (torch.rand(H, generator=g) + 0.5).half().cuda()
    offs = (0, kd, 2 * kd, conv_dim) + ((conv_dim + nv * dv, conv_dim + nv * dv + nv) if ab == "proj" else (-1, -1))
    lazy = lambda rows: K.lazy_norm(hres[rows], torch.cat([hres[rows].pow(2).sum(-1, keepdim=True), torch.zeros(len(rows), 3, device="cuda")], 1), wnorm)  # noqa: E731
    starts = [sum(sizes[:i]) for i in range(ns + 1)]
    parents = [_tree(n, kind) for n in sizes]
    paths, entries = [], []
    for s, par in enumerate(parents):
        up = []
        for t, q in enumerate(par):
            up.append((up[q] if q >= 0 else []) + [t])
            entries.append((s, 0, 0, 0, sum(1 << a for a in up[t])))
        paths += [(s, [starts[s] + a for a in u]) for u in up]
    rows, seq_rows = K.make_rows(entries, "cuda"), torch.tensor(starts, dtype=torch.int32, device="cuda")
    out = torch.zeros(R, nv * dv, dtype=torch.float16, device="cuda")
    p, st = L.DeltaParams(), L.SpecStage()
    p.proj, p.ld = proj.data_ptr(), ld
    p.off_q, p.off_k, p.off_v, p.off_z, p.off_a, p.off_b = offs
    p.xn, p.ldx, p.H, p.wa, p.wb = xn.data_ptr(), H, H, wa.data_ptr(), wb.data_ptr()
    every = list(range(R))
    keep = lazy(every) if ab == "lazy" else None
    if keep is not None:
        p.ln = keep
    p.conv_w, p.conv_state, p.state = conv_w.data_ptr(), conv.data_ptr(), state.data_ptr()
    p.A_log, p.dt_bias, p.norm_w = A_log.data_ptr(), dt_bias.data_ptr(), norm_w.data_ptr()
    p.seq_rows, p.rows, p.out, p.ldo = seq_rows.data_ptr(), rows.data_ptr(), out.data_ptr(), out.stride(0)
    p.nk, p.nv, p.n_seqs, p.eps = nk, nv, ns, 1e-6
    off = [C.c_int() for _ in range(4)]
    L.lib().b2_spec_stage_layout.restype = C.c_longlong
    blk = int(L.lib().b2_spec_stage_layout(nk, nv, dk, dv, *[C.byref(o) for o in off]))
    stage = torch.zeros(ns * blk, dtype=torch.uint8, device="cuda")
    st.base, st.seq_stride, st.layer_stride = stage.data_ptr(), blk, ns * blk
    st.off_k, st.off_u, st.off_g, st.off_x = (o.value for o in off)
    s0, c0 = state.clone(), conv.clone()
    L.check(L.lib().b2_deltanet_verify(C.byref(p), C.byref(st), 0, dk, dv, L.stream()), "verify")
    assert torch.equal(state, s0) and torch.equal(conv, c0)
    for r, (s, path) in enumerate(paths):
        one = torch.tensor([0, len(path)], dtype=torch.int32, device="cuda")
        ref = K.deltanet_step(proj[path].contiguous(), offs, conv_w, conv.clone(), state.clone(), A_log, dt_bias, norm_w,
                              K.make_rows([(s, 0, 0, 0, 1)] * len(path), "cuda"), one, nk, nv, dk, dv,
                              xn=xn[path].contiguous() if ab == "xn" else None, wa=wa if ab != "proj" else None,
                              wb=wb if ab != "proj" else None, ln=lazy(path) if ab == "lazy" else None)[-1]
        err = float((out[r].float() - ref.float()).abs().max() / ref.float().abs().max())
        assert err < 2e-3, (r, err)


class _Verify:
    """One launch of the verify kernel over chains of `n` drafts of `ns` sequences, heads of 64."""

    def __init__(self, nk=2, nv=4, ns=3, n=4, state_offset=0):
        from mi50grad_b200.ops import kernels as K
        g = torch.Generator().manual_seed(8)
        rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
        d, vd = 64, nv * 64
        self.cd = cd = 2 * nk * d + vd
        self.dims, self.offs = (nk, nv, d, d), (0, nk * d, 2 * nk * d, cd, cd + vd, cd + vd + nv)
        self.proj = rnd(ns * n, cd + vd + 2 * nv).half().cuda()
        self.w = [(rnd(cd, 4) * 0.3).half().cuda(), (torch.rand(nv, generator=g) * 1.5 - 1.0).cuda(), (rnd(nv) * 0.5).half().cuda(),
                  (torch.rand(d, generator=g) + 0.5).half().cuda()]
        self.conv = rnd(ns, nv, d // 32, 2 * d + 32, 3).half().cuda()
        self.state = torch.cat([torch.zeros(state_offset), (rnd(ns, nv, d, d) * 0.3).flatten()]).cuda()[state_offset:].view(ns, nv, d, d)
        self.rows = K.make_rows([(s, 0, 0, 0, (2 << i) - 1) for s in range(ns) for i in range(n)], "cuda")
        self.seq_rows = torch.arange(ns + 1, dtype=torch.int32, device="cuda") * n
        self.out, self.ns = torch.zeros(ns * n, vd, dtype=torch.float16, device="cuda"), ns

    def __call__(self):
        import ctypes as C
        from mi50grad_b200.ops import lib as L
        nk, nv, dk, dv = self.dims
        p, st = L.DeltaParams(), L.SpecStage()
        p.proj, p.ld = self.proj.data_ptr(), self.proj.stride(0)
        p.off_q, p.off_k, p.off_v, p.off_z, p.off_a, p.off_b = self.offs
        p.conv_w, p.A_log, p.dt_bias, p.norm_w = (t.data_ptr() for t in self.w)
        p.conv_state, p.state = self.conv.data_ptr(), self.state.data_ptr()
        p.seq_rows, p.rows, p.out, p.ldo = self.seq_rows.data_ptr(), self.rows.data_ptr(), self.out.data_ptr(), self.out.stride(0)
        p.nk, p.nv, p.n_seqs, p.eps = nk, nv, self.ns, 1e-6
        off = [C.c_int() for _ in range(4)]
        L.lib().b2_spec_stage_layout.restype = C.c_longlong
        blk = int(L.lib().b2_spec_stage_layout(nk, nv, dk, dv, *[C.byref(o) for o in off]))
        self.stage = torch.empty(self.ns * blk, dtype=torch.uint8, device="cuda")
        st.base, st.seq_stride, st.layer_stride = self.stage.data_ptr(), blk, self.ns * blk
        st.off_k, st.off_u, st.off_g, st.off_x = (o.value for o in off)
        L.check(L.lib().b2_deltanet_verify(C.byref(p), C.byref(st), 0, dk, dv, L.stream()), "verify")
        return self.out


def test_verify_of_states_off_the_16_byte_boundary():
    a, b = _Verify(), _Verify(state_offset=1)
    assert a.state.data_ptr() % 16 == 0 and b.state.data_ptr() % 16 == 4
    assert torch.equal(a(), b())


def test_verify_directly_after_the_step_that_left_its_states():
    """The verify kernel may begin under the step kernel before it; it reads the states that this leaves all the same."""
    from mi50grad_b200.ops import kernels as K
    v = _Verify()
    nk, nv, dk, dv = v.dims
    S0, c0, got = v.state.clone(), v.conv.clone(), []
    one = torch.arange(v.ns + 1, dtype=torch.int32, device="cuda")
    rows = K.make_rows([(s, 0, 0, 0, 1) for s in range(v.ns)], "cuda")
    for i in range(8):
        v.state.copy_(S0)
        v.conv.copy_(c0)
        for _ in range(3):
            K.deltanet_step(v.proj[:v.ns], v.offs, v.w[0], v.conv, v.state, *v.w[1:], rows, one, nk, nv, dk, dv)
        if i == 0:
            torch.cuda.synchronize()
        got.append(v().clone())
    assert all(torch.equal(g, got[0]) for g in got)
