"""What this engine is asked to do in use, as cases that can be timed and checked.

A case names a decoder (the hybrid decoder with INT4 weights, Degedra, Vekerax), one of the layer sizes that the
benchmark of this repository uses, and a call of the engine:

    generate   a prompt and some greedy tokens (`generate_tokens`)
    prompt     a prompt alone (`prefill_tokens`)
    decode     greedy steps from sequences that are there already: one sequence token by token from the host
               (`step_host`, the loop of the generation API), several in one batch (`decode_tokens`)
    verify     one draft-verification step of several sequences (`spec_step`)

Weights are random, with one thing that a trained model has and random weights have not: a sure next token.  The
output head of the hybrid decoder and of Degedra is the embedding moved by one token, so that the token after t is
t + 1 by a margin of many times any rounding; drafts can then be right or wrong on purpose, and greedy tokens do not
depend on the order of a sum.  (Vekerax ties its head to the embedding, which it scales by the root of the width:
there the token after t is t.)

`exact` is the same work in 64 bits, from the equations, in plain torch.
"""
import math

import torch

DEV = "cuda"

# width, feed-forward, attention heads / kv heads / dim, recurrence heads (of 64), window, layers
SIZES = {
    "2k": (2048, 6144, 16, 4, 128, 32, 1024, 12),
    "4k": (4096, 12288, 32, 8, 128, 64, 1024, 8),
    "5k": (5120, 17408, 40, 8, 128, 80, 4096, 6),
}
VOCAB = 65536
EPS = 1e-5
DRAFT = 4


def listed():
    return [
        # the smallest call: a four-layer model of width 256, where launches and latencies are all there is
        dict(name="tiny hybrid: generate", model="hybrid", size="tiny", op="generate", tokens=16, new=8, batch=1, ctx=0, form="int4"),
        # one user who is answered: 27B, INT4 weights, a short context (the headline benchmark)
        dict(name="27b: decode", model="hybrid", size="27b", op="decode", tokens=0, new=8, batch=1, ctx=133, form="int4"),
        # the prompt of the headline benchmark
        dict(name="27b: prompt of 512", model="hybrid", size="27b", op="prompt", tokens=512, new=0, batch=1, ctx=0, form="int4"),
        # a busy server: 16 sequences of about 4000 tokens, four drafted tokens each, half of them right
        dict(name="27b: verify 16 drafts", model="hybrid", size="27b", op="verify", tokens=0, new=1, batch=16, ctx=4051, form="int4"),
        # the published checkpoint's form: attention and recurrence weights in fp16; a few users, long contexts
        dict(name="hybrid 5k fp16: decode 5", model="hybrid", size="5k", op="decode", tokens=0, new=8, batch=5, ctx=7001, form="fp16"),
        # a batch too large for the few-row kernels
        dict(name="hybrid 2k: decode 24", model="hybrid", size="2k", op="decode", tokens=0, new=4, batch=24, ctx=700, form="int4"),
        # a chat turn
        dict(name="hybrid 4k: prompt of 77", model="hybrid", size="4k", op="prompt", tokens=77, new=0, batch=1, ctx=0, form="int4"),
        # a document
        dict(name="hybrid 4k: prompt of 3001", model="hybrid", size="4k", op="prompt", tokens=3001, new=0, batch=1, ctx=0, form="int4"),
        # the dense-weight decoders: a user who is answered, a prompt, everything in 32 bits, a small batch
        dict(name="degedra 4k: decode", model="degedra", size="4k", op="decode", tokens=0, new=8, batch=1, ctx=1500, form="bf16"),
        dict(name="degedra 5k: prompt of 1000", model="degedra", size="5k", op="prompt", tokens=1000, new=0, batch=1, ctx=0, form="bf16"),
        dict(name="degedra 2k fp32: prompt of 200", model="degedra", size="2k", op="prompt", tokens=200, new=0, batch=1, ctx=0, form="fp32"),
        dict(name="vekerax 4k: generate", model="vekerax", size="4k", op="generate", tokens=300, new=16, batch=1, ctx=0, form="bf16"),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    model = rng.choice(["hybrid"] * 4 + ["degedra", "degedra", "vekerax"])
    size = rng.choice(["2k", "4k", "5k"] + (["27b", "tiny"] if model == "hybrid" else []))
    op = rng.choice(["generate", "prompt", "decode", "decode"] + (["verify"] if model == "hybrid" else []))
    c = dict(model=model, size=size, op=op, tokens=0, new=0, batch=1, ctx=0, form="int4" if model == "hybrid" else "bf16")
    big = size == "27b"
    if op in ("generate", "prompt"):
        c["tokens"] = log(9, 512 if big else 3000)
        c["new"] = log(2, 8 if big else 16) if op == "generate" else 0
    elif op == "decode":
        c["batch"] = 1 if rng.random() < 0.5 else log(2, 32 if model == "hybrid" else 8)
        c["ctx"] = log(30, 2000 if big else 8000)
        c["new"] = log(2, 8)
    else:
        c["batch"], c["new"], c["ctx"] = log(1, 16), 1, log(100, 4051)
    if model == "hybrid" and size != "tiny" and op == "decode" and c["batch"] <= 8 and rng.random() < 0.3:
        c["form"] = "fp16"
    if model == "degedra" and size == "2k" and c["tokens"] <= 512 and rng.random() < 0.3:
        c["form"] = "fp32"
    return c


# ---------------------------------------------------------------------------- sizes and weights

def _hybrid_dims(size):
    if size == "tiny":
        return dict(hidden_size=256, intermediate_size=704, num_hidden_layers=4, vocab_size=1024, num_attention_heads=4,
                    num_key_value_heads=2, head_dim=64, linear_num_value_heads=4, linear_num_key_heads=2, linear_key_head_dim=64,
                    linear_value_head_dim=64, full_attention_interval=4, rms_norm_eps=1e-6)
    if size == "27b":
        return dict(hidden_size=5120, intermediate_size=17408, num_hidden_layers=64, vocab_size=248320, num_attention_heads=24,
                    num_key_value_heads=4, head_dim=256, linear_num_value_heads=48, linear_num_key_heads=16, linear_key_head_dim=128,
                    linear_value_head_dim=128, full_attention_interval=4, rms_norm_eps=1e-6)
    w, ff, h, kv, d, sh, _, n = SIZES[size]
    return dict(hidden_size=w, intermediate_size=ff, num_hidden_layers=n, vocab_size=VOCAB, num_attention_heads=h * d // 256,
                num_key_value_heads=max(1, kv * d // 256), head_dim=256, linear_num_value_heads=sh // 2, linear_num_key_heads=sh // 4,
                linear_key_head_dim=128, linear_value_head_dim=128, full_attention_interval=2, rms_norm_eps=1e-6)


def _is_full(c, i):
    return (i + 1) % c["full_attention_interval"] == 0


def _dims(case):
    """(width, feed-forward, layers, vocabulary)"""
    if case["model"] == "hybrid":
        c = _hybrid_dims(case["size"])
        return c["hidden_size"], c["intermediate_size"], c["num_hidden_layers"], c["vocab_size"]
    w, ff, *_, n = SIZES[case["size"]]
    return w, ff, n, VOCAB


class _Random:
    """Values on the GPU from a seed and a place."""

    def __init__(self, seed, place):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(1000003 * seed + place)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float16):
        t = torch.empty(*shape, dtype=torch.float32 if math.prod(shape) < 1 << 26 else dtype, device=DEV)
        return t.normal_(mean, std, generator=self.g).to(dtype)

    def uniform(self, lo, hi, *shape):
        return torch.empty(*shape, device=DEV).uniform_(lo, hi, generator=self.g)

    def int4(self, K, N):
        """(nibbles [K/8, N], scales, zero points [K/128, N]) as a GPTQ checkpoint has them.  Nibbles are uniform and
        zero points 7 or 8, so that no column leans to one side on the whole: with 8 alone every output has the same
        small offset, which 64 layers amplify until the logits no longer depend on the tokens."""
        q = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), dtype=torch.int32, device=DEV, generator=self.g)
        s = self.uniform(0.002, 0.02, -(-K // 128), N)
        z = torch.randint(7, 9, s.shape, device=DEV, generator=self.g)
        return q, s.half(), z.half()


# name -> (outputs, inputs) of a hybrid layer's projections; those in ALWAYS_INT4 have INT4 weights in every form
ALWAYS_INT4 = ("gate", "up", "down")
ALWAYS_FP16 = ("la_a", "la_b")


def _hybrid_shapes(c, full):
    h, f = c["hidden_size"], c["intermediate_size"]
    if full:
        qd, kd = c["num_attention_heads"] * c["head_dim"], c["num_key_value_heads"] * c["head_dim"]
        s = dict(q=(qd, h), q_gate=(qd, h), k=(kd, h), v=(kd, h), o=(h, qd))
    else:
        nv = c["linear_num_value_heads"]
        kd, vd = c["linear_num_key_heads"] * c["linear_key_head_dim"], nv * c["linear_value_head_dim"]
        s = dict(la_qkv=(2 * kd + vd, h), la_a=(nv, h), la_b=(nv, h), la_z=(vd, h), la_out=(h, vd))
    return dict(s, gate=(f, h), up=(f, h), down=(h, f))


def _hybrid_layer(case, c, i, seed):
    """name -> (nibbles, scales, zero points) or a tensor"""
    r, full = _Random(seed, i), _is_full(c, i)
    w = {}
    for n, (out, k) in _hybrid_shapes(c, full).items():
        four = n not in ALWAYS_FP16 and (case["form"] == "int4" or n in ALWAYS_INT4)
        w[n] = r.int4(k, out) if four else r.normal(out, k, std=0.02)
    norm = lambda n: r.normal(n, std=0.1, mean=1.0)  # noqa: E731
    w["attn_norm"], w["ffn_norm"] = norm(c["hidden_size"]), norm(c["hidden_size"])
    if full:
        w["q_norm"], w["k_norm"] = norm(c["head_dim"]), norm(c["head_dim"])
    else:
        nv = c["linear_num_value_heads"]
        w["la_conv1d"] = r.normal(_hybrid_shapes(c, False)["la_qkv"][0], 4, std=0.3)
        w["la_A_log"] = r.uniform(-1.0, 0.5, nv)
        w["la_dt_bias"], w["la_norm"] = r.normal(nv, std=0.5), norm(c["linear_value_head_dim"])
    return w


# standard deviation of the embedding: a fifth of the residual stream's in the end (a half of it for the tiny model)
EMBED_STD = {"tiny": 2.0, "2k": 12.0, "4k": 25.0, "5k": 40.0, "27b": 110.0}


def _hybrid_ends(case, seed):
    c = _hybrid_dims(case["size"])
    r, std = _Random(seed, 999), EMBED_STD[case["size"]]
    embed = r.normal(c["vocab_size"], c["hidden_size"], std=std)
    return embed, torch.roll(embed, 1, 0).mul_(0.05 / std), r.normal(c["hidden_size"], std=0.1, mean=1.0)


def _mixer_config(case):
    from mi50grad_b200.config import (DegedraConfig, LightningSpec, ParallelLayerSpec, SSDSpec, StreamLayerSpec, VekeraxConfig,
                                      WindowAttentionSpec)
    w, ff, h, kv, d, sh, win, n = SIZES[case["size"]]
    if case["model"] == "degedra":
        layer = ParallelLayerSpec(WindowAttentionSpec(h, kv, d, d, 1e6, d ** -0.5, win), SSDSpec(sh, 64, 128, 8, 4, 8), 0.7, 1.0, ff)
        return DegedraConfig(w, VOCAB, EPS, [layer] * n, 30.0)
    att = StreamLayerSpec(WindowAttentionSpec(h, kv, d, 0, 0.0, d ** -0.5, win, vdim=d, head_norm=True, keep_first=4, softcap=30.0, sink=True), ff)
    rec = StreamLayerSpec(LightningSpec(sh // 2, 128, 128, _decays(sh // 2)), ff)
    return VekeraxConfig(w, VOCAB, EPS, [att if i % 2 == 0 else rec for i in range(n)], w ** 0.5, 1.0, 4)


def _decays(heads):
    return tuple(1.0 - 2.0 ** (-1 - 4 * i / heads) for i in range(heads))


def _mixer_layer(case, i, seed):
    w, ff, h, kv, d, sh, _, _ = SIZES[case["size"]]
    if case["model"] == "degedra":
        ch = sh * 64 + 2 * 8 * 128
        s = dict(norm1=(w,), q=(h * d, w), k=(kv * d, w), q_norm=(h * d,), k_norm=(kv * d,), attn_o=(w, h * d),
                 ssd_in=(sh * 64 + ch + sh, w), conv=(ch, 4), conv_b=(ch,), dt_bias=(sh,), A_log=(sh,), D=(sh,), ssd_norm=(sh * 64,), ssd_o=(w, sh * 64))
    elif i % 2 == 0:
        s = dict(q=(h * d, w), k=(kv * d, w), v=(kv * d, w), o=(w, h * d), q_norm=(d,), k_norm=(d,), sink=(h,), norm1=(w,))
    else:
        e = sh // 2 * 128
        s = dict(q=(e, w), k=(e, w), v=(e, w), g=(e, w), o=(w, e), out_norm=(e,), norm1=(w,))
    s.update(norm2=(w,), gate=(ff, w), up=(ff, w), down=(w, ff))
    if case["model"] == "vekerax":
        for q in (1, 2):
            s.update({"hc%d_in" % q: (4,), "hc%d_out" % q: (4,), "hc%d_mix" % q: (4, 4)})
    r, t, bf = _Random(seed, i), {}, torch.bfloat16
    for n, sh_ in s.items():
        if "norm" in n:
            t[n] = r.normal(*sh_, std=0.1, mean=1.0, dtype=bf)
        elif n == "dt_bias":
            t[n] = r.normal(*sh_, std=0.7, mean=-2.0, dtype=bf)
        elif n == "A_log":
            t[n] = r.uniform(0.0, 2.5, *sh_).to(bf)
        elif n == "D":
            t[n] = r.normal(*sh_, std=0.3, mean=1.0, dtype=bf)
        elif n == "conv_b":
            t[n] = r.normal(*sh_, std=0.2, dtype=bf)
        elif n == "sink":
            t[n] = r.normal(*sh_, dtype=bf)
        elif n.endswith("_mix"):
            t[n] = (0.95 * torch.eye(4, device=DEV) + r.normal(4, 4, std=0.075, dtype=torch.float32)).to(bf)
        elif n.startswith("hc"):
            m = 0.25 if n.endswith("_in") else 1.0
            t[n] = r.normal(*sh_, std=0.3 * m, mean=m, dtype=bf)
        else:
            t[n] = r.normal(*sh_, std=sh_[1] ** -0.5, dtype=bf)
    return t


def _mixer_ends(case, seed):
    w, r, bf = SIZES[case["size"]][0], _Random(seed, 999), torch.bfloat16
    tied = case["model"] == "vekerax"
    embed = r.normal(VOCAB, w, std=w ** -0.5 if tied else 1.0, dtype=bf)
    return embed, embed if tied else torch.roll(embed, 1, 0).mul_(2 * w ** -0.5), r.normal(w, std=0.1, mean=1.0, dtype=bf)


# ---------------------------------------------------------------------------- sequences

def _contexts(case):
    """Lengths of the sequences that are there before the call: no two alike."""
    return [max(1, case["ctx"] - 7 * b * max(1, case["ctx"] // 200)) for b in range(case["batch"])]


def _tokens(case, seed):
    """The prompt, or the pending token of every sequence."""
    g = torch.Generator().manual_seed(seed + 17)
    return torch.randint(0, _dims(case)[3] - 64, (max(case["tokens"], case["batch"]),), generator=g).tolist()


def _draft(case, tok):
    """Four tokens after `tok`: two that the model will say itself, then two that it will not."""
    return [tok + 1, tok + 2, tok + 30, tok + 31]


def _history(case, seed):
    """Per sequence: a dict of what its cache and state hold, as `state_dict` gives it, and for the hybrid decoder the
    convolution's last inputs [layers, channels, 3] as well."""
    out = []
    for b, n in enumerate(_contexts(case) if case["ctx"] else []):
        r = _Random(seed, 2000 + b)
        if case["model"] == "hybrid":
            c = _hybrid_dims(case["size"])
            full = sum(_is_full(c, i) for i in range(c["num_hidden_layers"]))
            lin = c["num_hidden_layers"] - full
            nk, nv, dk, dv = c["linear_num_key_heads"], c["linear_num_value_heads"], c["linear_key_head_dim"], c["linear_value_head_dim"]
            kv = (full, n, c["num_key_value_heads"], c["head_dim"])
            taps = r.normal(lin, 2 * nk * dk + nv * dv, 3, std=2.0)
            out.append(dict(k=r.normal(*kv), v=r.normal(*kv, std=2.0), S=r.normal(lin, nv, dk, dv, std=0.3, dtype=torch.float32),
                            taps=taps, conv=_by_block(taps, nk, nv, dk, dv)))
            continue
        w, ff, h, kv, d, sh, _, layers = SIZES[case["size"]]
        t = torch.float32 if case["form"] == "fp32" else torch.bfloat16
        s = {}
        for i in range(layers):
            att = case["model"] == "degedra" or i % 2 == 0
            rec = case["model"] == "degedra" or i % 2 == 1
            heads, state, vdim = ((sh, 128, 64) if case["model"] == "degedra" else (sh // 2, 128, 128)) if rec else (0, 1, 1)
            s["k%d" % i] = r.normal(n, kv if att else 0, d if att else 8, dtype=t)
            s["v%d" % i] = r.normal(n, kv if att else 0, d if att else 8, dtype=t)
            s["S%d" % i] = r.normal(heads, state, vdim, std=0.5, dtype=torch.float32)
            ch = sh * 64 + 2 * 8 * 128 if case["model"] == "degedra" else 0
            s["conv%d" % i] = r.normal(3 if ch else 0, ch, dtype=t)
        out.append(s)
    return out


def _by_block(taps, nk, nv, dk, dv):
    """The convolution's inputs as the states keep them: every value head has a copy for each 32 of its columns,
    of its key head's q and k channels and of those 32: [layers][value heads][dv / 32][2 dk + 32][3]."""
    lin = taps.shape[0]
    q = taps[:, :nk * dk].reshape(lin, nk, 1, dk, 3).repeat_interleave(nv // nk, 1).expand(-1, -1, dv // 32, -1, -1)
    k = taps[:, nk * dk:2 * nk * dk].reshape(lin, nk, 1, dk, 3).repeat_interleave(nv // nk, 1).expand(-1, -1, dv // 32, -1, -1)
    v = taps[:, 2 * nk * dk:].reshape(lin, nv, dv // 32, 32, 3)
    return torch.cat([q, k, v], 3)


# ---------------------------------------------------------------------------- the engine

def _engine(case, seed):
    top = max(case["ctx"], case["tokens"]) + case["new"] + 64
    if case["model"] == "hybrid":
        from mi50grad_b200.config import EngineConfig, QwenConfig
        from mi50grad_b200.engine.engine import InferenceEngine
        from mi50grad_b200.models.weights import LayerWeights
        from mi50grad_b200.utils.quant import DenseLinear, Int4Linear
        c = _hybrid_dims(case["size"])
        cfg = QwenConfig(attn_quantized=case["form"] == "int4", **c)
        eng = InferenceEngine(cfg, max_seq_len=top, max_batch=case["batch"],
                              engine_config=EngineConfig(max_step_rows=max(8, case["batch"] * (DRAFT + 1))))
        lin = lambda w: Int4Linear(*w) if isinstance(w, tuple) else DenseLinear(w)  # noqa: E731
        for i in range(cfg.num_hidden_layers):
            w = _hybrid_layer(case, c, i, seed)
            names = _hybrid_shapes(c, _is_full(c, i))
            eng.load_layer_weights(i, LayerWeights("full_attention" if _is_full(c, i) else "linear_attention",
                                                   **{n: lin(t) if n in names else t for n, t in w.items()}))
        embed, head, norm = _hybrid_ends(case, seed)
    else:
        from mi50grad_b200.config import EngineConfig
        if case["model"] == "degedra":
            from mi50grad_b200.engine.mixer_engine import MixerEngine as Engine
        else:
            from mi50grad_b200.engine.vekerax_engine import VekeraxEngine as Engine
        cfg = _mixer_config(case)
        eng = Engine(cfg, max_seq_len=top, max_batch=case["batch"], dtype="float32" if case["form"] == "fp32" else "bfloat16",
                     engine_config=EngineConfig(max_step_rows=64))
        for i in range(cfg.num_hidden_layers):
            eng.load_layer_weights(i, _mixer_layer(case, i, seed))
        embed, head, norm = _mixer_ends(case, seed)
    eng.load_embedding(embed)
    if case["model"] != "vekerax":
        eng.load_lm_head(head)
    eng.load_final_norm(norm)
    eng.build_decode_launch_cache()
    return eng


def prepare(case, seed):
    """An engine with its weights and, for steps of sequences that are there, their caches and states."""
    eng = _engine(case, seed)
    toks = _tokens(case, seed)
    st = dict(case=case, eng=eng, tokens=toks[:case["tokens"]] if case["tokens"] else toks[:case["batch"]], ctx=_contexts(case))
    for b, h in enumerate(_history(case, seed)):
        h.pop("taps", None)
        eng.states.load_state_dict(dict(h, length=torch.tensor(st["ctx"][b]), token=torch.tensor(toks[b])), b)
    st["seqs"] = eng.states.seqs.clone()
    if case["op"] == "verify":
        st["drafts"] = [_draft(case, t) for t in st["tokens"]]
        st["parents"] = [list(range(-1, DRAFT - 1))] * case["batch"]
    return st


def run(st):
    """One call, and what it leaves: tokens, logits, the cache rows that it wrote, recurrent states."""
    case, eng, toks = st["case"], st["eng"], st["tokens"]
    op, n, batch = case["op"], case["new"], case["batch"]
    wrote = [(0, 0)]
    if op == "generate":
        got = torch.tensor(eng.generate_tokens(toks, n))
        wrote = [(0, len(toks) + n - 1)]
    elif op == "prompt":
        eng.reset(0)
        got = torch.tensor([eng.prefill_tokens(toks, 0)])
        wrote = [(0, len(toks))]
    else:
        # the sequences start where they did the last time (one small copy); the recurrent states go on
        eng.states.seqs.copy_(st["seqs"])
        if op == "verify":
            res = eng.spec_step(st["drafts"], st["parents"], list(range(batch)), toks, graph=True)
            got = torch.tensor([list(a) + [nxt] for a, nxt in res])
            wrote = [(c, c + got.shape[1]) for c in st["ctx"]]
        elif batch == 1:
            t, out = toks[0], []
            for _ in range(n):
                t = eng.step_host(t, 0)
                out.append(t)
            got = torch.tensor(out)
            wrote = [(st["ctx"][0], st["ctx"][0] + n)]
        else:
            got = eng.decode_tokens(n, list(range(batch)))
            wrote = [(c, c + n) for c in st["ctx"]]
    rows = batch * (DRAFT + 1) if op == "verify" else batch
    many = rows > eng.max_rows
    logits = eng.buf["p_logits" if many else "logits"][:rows, :eng.config.vocab_size]
    s = eng.states
    if case["model"] == "hybrid":
        return dict(tokens=got, logits=logits, S=s.dn.S[:, :batch], conv=s.dn.conv[:, :batch],
                    k=[s.kv.k[:, b, i:j] for b, (i, j) in enumerate(wrote)], v=[s.kv.v[:, b, i:j] for b, (i, j) in enumerate(wrote)])
    i, j = min(w[0] for w in wrote), max(w[1] for w in wrote)
    some = lambda ts: [t[:, i:j] for t in ts if t.numel()]  # noqa: E731
    return dict(tokens=got, logits=logits, S=[t for t in s.S if t.numel()], conv=[t for t in s.conv if t.numel()], k=some(s.k), v=some(s.v))


def _params(case):
    """(bytes of the projections and the head, multiply-adds per row of the layers' projections)"""
    w, ff, n, vocab = _dims(case)
    if case["model"] == "hybrid":
        c, by, ops = _hybrid_dims(case["size"]), 0.0, 0.0
        for i in range(n):
            for name, (o, k) in _hybrid_shapes(c, _is_full(c, i)).items():
                four = name not in ALWAYS_FP16 and (case["form"] == "int4" or name in ALWAYS_INT4)
                by += o * k * (0.5 + 4 / 128 if four else 2)
                ops += o * k
        return by + 2.0 * vocab * w, ops
    _, _, h, kv, d, sh, _, _ = SIZES[case["size"]]
    ops = 3 * w * ff * n
    if case["model"] == "degedra":
        ops += n * w * (2 * h * d + kv * d + sh * 64 * 3 + 2 * 8 * 128 + sh)
    else:
        ops += (n + 1) // 2 * w * (2 * h * d + 2 * kv * d) + n // 2 * w * 5 * (sh // 2 * 128)
    return (4 if case["form"] == "fp32" else 2) * float(ops + vocab * w), float(ops)


def _per_token(case):
    """(bytes of a cached token over all layers, bytes of a sequence's recurrent states, window, attention columns over all layers)"""
    n = _dims(case)[2]
    if case["model"] == "hybrid":
        c = _hybrid_dims(case["size"])
        full = sum(_is_full(c, i) for i in range(n))
        return (full * 4 * c["num_key_value_heads"] * c["head_dim"],
                (n - full) * 4 * c["linear_num_value_heads"] * c["linear_key_head_dim"] * c["linear_value_head_dim"], 1 << 30,
                full * c["num_attention_heads"] * c["head_dim"])
    _, _, h, kv, d, sh, win, _ = SIZES[case["size"]]
    e = 4 if case["form"] == "fp32" else 2
    att, rec = (n, n) if case["model"] == "degedra" else ((n + 1) // 2, n // 2)
    return att * 2 * kv * d * e, rec * 4 * sh * 64 * 128, win, att * h * d


def work(case):
    """Weights once for every step that needs them (a prompt is one), cached rows that a step can see, recurrent states in
    and out, logits out."""
    by, ops = _params(case)
    w, _, _, vocab = _dims(case)
    token, state, win, cols = _per_token(case)
    op, batch, new = case["op"], case["batch"], case["new"]
    head = float(vocab * w)
    if op in ("prompt", "generate"):
        t, steps = case["tokens"], max(0, new - 1)
        seen = sum(min(i + 1, win) for i in range(t)) + steps * min(t, win)
        return {"bytes": by * (1 + steps) + token * (t + steps * min(t, win)) + state * (1 + 2 * steps) + 4 * vocab * (1 + steps),
                "flops": 2 * ops * (t + steps) + 2 * head * (1 + steps) + 4 * cols * seen}
    rows, steps = (batch * (DRAFT + 1), 1) if op == "verify" else (batch, new)
    seen = sum(min(c, win) for c in _contexts(case))
    return {"bytes": steps * (by + token * seen + 2 * state * batch + 4 * vocab * rows),
            "flops": steps * (2 * ops * rows + 2 * head * rows + 4 * cols * seen * rows / batch)}


def tolerance(case):
    """About four times the distance from the result in 64 bits, which is what rounding activations to fp16 (bf16: 8 times
    coarser; it is cut to 0.03) after every product leaves behind; the deepest model adds up the most of it.  Measured:
    2.8e-3 for 64 layers, 1.3e-3 for 6 to 12, 1.9e-2 in bf16, 1.4e-5 in fp32."""
    if case["form"] == "fp32":
        return {"rel": 6e-5}
    if case["form"] == "bf16":
        return {"rel": 0.03}
    return {"rel": 0.011 if case["size"] == "27b" else 0.006}


# ---------------------------------------------------------------------------- the same in 64 bits

F64 = torch.float64


def _dense64(w):
    """[K, N] in 64 bits of (nibbles, scales, zero points), or the transpose of [N, K]"""
    if not isinstance(w, tuple):
        return w.to(F64).t()
    q, s, z = (t.to(F64) if t.is_floating_point() else t for t in w)
    K, N = q.shape[0] * 8, q.shape[1]
    nib = torch.stack([(q >> (4 * j)) & 15 for j in range(8)], 1).reshape(K, N)
    wide = lambda t: t.repeat_interleave(128, 0)[:K]  # noqa: E731
    return (nib - wide(z)) * wide(s)


def _mm(x, w):
    return x @ _dense64(w)


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _soft_plus(x):
    return torch.clamp(x, min=0) + torch.log1p(torch.exp(-x.abs()))


def _turn(x, pos, dims, base, pairs):
    """Rotary positions over the first `dims` of every head: pairs (2i, 2i + 1), or (i, i + dims / 2)."""
    h = dims // 2
    f = float(base) ** (-2.0 * torch.arange(h, dtype=F64, device=x.device) / dims)
    a = pos.to(F64)[:, None] * f
    c, s = torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]
    u, v = (x[..., 0:dims:2], x[..., 1:dims:2]) if pairs else (x[..., :h], x[..., h:dims])
    y, z = u * c - v * s, u * s + v * c
    return torch.cat([torch.stack([y, z], -1).flatten(-2) if pairs else torch.cat([y, z], -1), x[..., dims:]], -1)


def _attend(q, k, v, scale, first, window=0, keep=0, cap=0.0, sink=None):
    """q [n, H, d] at positions first ..; k, v [m, G, *] at positions 0 .. : causal attention in rows of at most 256 queries"""
    n, H, _ = q.shape
    m, G, _ = k.shape
    out = []
    j = torch.arange(m, device=q.device)
    for a in range(0, n, 256):
        i = torch.arange(first + a, first + min(n, a + 256), device=q.device)[:, None]
        see = j <= i
        if window:
            see &= (i - j < window) | (j < keep)
        s = torch.einsum("nghd,mgd->ghnm", q[a:a + 256].reshape(-1, G, H // G, q.shape[-1]), k) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~see, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.to(F64).reshape(G, H // G, 1, 1).expand(-1, -1, s.shape[2], 1)], -1)
        p = torch.softmax(s, -1)[..., :m]
        out.append(torch.einsum("ghnm,mge->nghe", p, v).reshape(-1, H, v.shape[-1]))
    return torch.cat(out)


def _convolve(x, before, w, b=None):
    """x [n, channels] after `before` [taps - 1, channels] -> (SiLU of the causal convolution, all inputs)"""
    full = torch.cat([before, x])
    t = w.shape[1]
    y = sum(w[:, j].to(F64) * full[j:j + x.shape[0]] for j in range(t))
    return _silu(y if b is None else y + b.to(F64)), full


class _Sequence:
    """One sequence: the rows to feed, how many of them it keeps, and what it holds."""

    def __init__(self, tokens, keep, length, mem):
        self.tokens, self.keep, self.n0, self.mem = tokens, keep, length, mem


def _spans(seqs):
    a = 0
    for s in seqs:
        yield s, slice(a, a + len(s.tokens))
        a += len(s.tokens)


def _hybrid64(case, seed, seqs):
    """Runs the sequences' rows through the model: logits of all rows of the last layer as a function of a row list."""
    c = _hybrid_dims(case["size"])
    eps, hd, dk, dv = c["rms_norm_eps"], c["head_dim"], c["linear_key_head_dim"], c["linear_value_head_dim"]
    nq, nkv, nk, nv = c["num_attention_heads"], c["num_key_value_heads"], c["linear_num_key_heads"], c["linear_num_value_heads"]
    embed, head, norm = _hybrid_ends(case, seed)
    x = embed[torch.tensor([t for s in seqs for t in s.tokens], device=DEV)].to(F64)
    del embed
    jf = jl = 0
    for i in range(c["num_hidden_layers"]):
        w = _hybrid_layer(case, c, i, seed)
        xn = _rms(x, eps) * w["attn_norm"].to(F64)
        mixed = torch.empty(x.shape[0], nq * hd if _is_full(c, i) else nv * dv, dtype=F64, device=DEV)
        if _is_full(c, i):
            q, g, k, v = (_mm(xn, w[n]) for n in ("q", "q_gate", "k", "v"))
            for s, at in _spans(seqs):
                n = len(s.tokens)
                pos = torch.arange(s.n0, s.n0 + n, device=DEV)
                # a quarter of every head turns
                turn = lambda t, nw, m: _turn(_rms(t[at].reshape(n, m, hd), eps) * nw.to(F64), pos, hd // 4, 1e7, True)  # noqa: E731
                kk, vv = turn(k, w["k_norm"], nkv), v[at].reshape(n, nkv, hd)
                s.mem.setdefault("new_k", []).append(kk[:s.keep])
                s.mem.setdefault("new_v", []).append(vv[:s.keep])
                if s.n0:
                    kk, vv = torch.cat([s.mem["k"][jf].to(F64), kk]), torch.cat([s.mem["v"][jf].to(F64), vv])
                o = _attend(turn(q, w["q_norm"], nq), kk, vv, hd ** -0.5, s.n0)
                mixed[at] = o.reshape(n, -1) * torch.sigmoid(g[at])
            x = x + _mm(mixed, w["o"])
            jf += 1
        else:
            qkv, z, a, b = (_mm(xn, w[n]) for n in ("la_qkv", "la_z", "la_a", "la_b"))
            decay = torch.exp((-torch.exp(w["la_A_log"].to(F64)) * _soft_plus(a + w["la_dt_bias"].to(F64))).clamp(-20.0, 0.0))
            beta = torch.sigmoid(b)
            unit = lambda t: t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
            for s, at in _spans(seqs):
                n = len(s.tokens)
                before = s.mem["taps"][jl].to(F64).t() if s.n0 else torch.zeros(3, qkv.shape[1], dtype=F64, device=DEV)
                y, full = _convolve(qkv[at], before, w["la_conv1d"])
                qq = unit(y[:, :nk * dk].reshape(n, nk, dk)).repeat_interleave(nv // nk, 1) * dk ** -0.5
                kk = unit(y[:, nk * dk:2 * nk * dk].reshape(n, nk, dk)).repeat_interleave(nv // nk, 1)
                vv = y[:, 2 * nk * dk:].reshape(n, nv, dv)
                S = s.mem["S"][jl].to(F64).clone() if s.n0 else torch.zeros(nv, dk, dv, dtype=F64, device=DEV)
                out, dec, bet = torch.empty(n, nv, dv, dtype=F64, device=DEV), decay[at], beta[at]
                for t in range(n):
                    S *= dec[t][:, None, None]
                    d = (vv[t] - torch.bmm(kk[t][:, None], S)[:, 0]) * bet[t][:, None]
                    S.baddbmm_(kk[t][:, :, None], d[:, None])
                    out[t] = torch.bmm(qq[t][:, None], S)[:, 0]
                    if t + 1 == s.keep:
                        s.mem.setdefault("new_S", []).append(S.clone())
                s.mem.setdefault("new_taps", []).append(full[s.keep:s.keep + 3].t())
                o = _rms(out, 1e-6) * w["la_norm"].to(F64)
                mixed[at] = o.reshape(n, -1) * _silu(z[at])
            x = x + _mm(mixed, w["la_out"])
            jl += 1
        xn = _rms(x, eps) * w["ffn_norm"].to(F64)
        x = x + _mm(_silu(_mm(xn, w["gate"])) * _mm(xn, w["up"]), w["down"])
    xn = _rms(x, eps) * norm.to(F64)
    return lambda rows: torch.cat([xn[rows] @ head[a:a + 16384].to(F64).t() for a in range(0, head.shape[0], 16384)], 1)


def _mixer64(case, seed, seqs):
    width, ff, h, kv, d, sh, win, layers = SIZES[case["size"]]
    embed, head, norm = _mixer_ends(case, seed)
    x = embed[torch.tensor([t for s in seqs for t in s.tokens], device=DEV)].to(F64)
    two = case["model"] == "vekerax"
    if two:
        x = x * width ** 0.5
    xs = torch.stack([x] * 4) if two else None

    def attention(i, s, q, k, v, **more):
        s.mem["new_k%d" % i], s.mem["new_v%d" % i] = k, v
        if s.n0:
            k, v = torch.cat([s.mem["k%d" % i].to(F64), k]), torch.cat([s.mem["v%d" % i].to(F64), v])
        return _attend(q, k, v, d ** -0.5, s.n0, win, **more).reshape(q.shape[0], -1)

    def recurrence(i, s, q, k, v, decay):
        """q, k [n, heads, state], v [n, heads, vdim], decay [n, heads]"""
        S = s.mem["S%d" % i].to(F64).clone() if s.n0 else torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F64, device=DEV)
        out = torch.empty_like(v)
        for t in range(q.shape[0]):
            S *= decay[t][:, None, None]
            S.baddbmm_(k[t][:, :, None], v[t][:, None])
            out[t] = torch.bmm(q[t][:, None], S)[:, 0]
        s.mem["new_S%d" % i] = S
        return out

    def parallel(i, w, x):
        """attention beside a Mamba-2 recurrence"""
        inner, ch = sh * 64, sh * 64 + 2 * 8 * 128
        q, k, u = (_mm(x, w[n]) for n in ("q", "k", "ssd_in"))
        left, right = torch.empty(x.shape[0], h * d, dtype=F64, device=DEV), torch.empty(x.shape[0], inner, dtype=F64, device=DEV)
        for s, at in _spans(seqs):
            n = len(s.tokens)
            pos = torch.arange(s.n0, s.n0 + n, device=DEV)
            turn = lambda t, nw: _turn((_rms(t[at], EPS) * w[nw].to(F64)).reshape(n, -1, d), pos, d, 1e6, False)  # noqa: E731
            left[at] = attention(i, s, turn(q, "q_norm"), turn(k, "k_norm"), k[at].reshape(n, kv, d))
            z, xbc, dt = u[at][:, :inner], u[at][:, inner:inner + ch], u[at][:, inner + ch:]
            before = s.mem["conv%d" % i].to(F64) if s.n0 else torch.zeros(3, ch, dtype=F64, device=DEV)
            y, full = _convolve(xbc, before, w["conv"], w["conv_b"])
            s.mem["new_conv%d" % i] = full[-3:]
            dt = _soft_plus(dt + w["dt_bias"].to(F64))
            group = lambda t: t.reshape(n, 8, 128).repeat_interleave(sh // 8, 1)  # noqa: E731
            xh = y[:, :inner].reshape(n, sh, 64)
            o = recurrence(i, s, group(y[:, inner + 1024:]), group(y[:, inner:inner + 1024]), dt[:, :, None] * xh,
                           torch.exp(-torch.exp(w["A_log"].to(F64)) * dt))
            o = (o + w["D"].to(F64)[:, None] * xh).reshape(n, inner) * _silu(z)
            right[at] = _rms(o.reshape(n, 8, inner // 8), EPS).reshape(n, inner) * w["ssd_norm"].to(F64)
        return 0.7 * _mm(left, w["attn_o"]) + _mm(right, w["ssd_o"])

    def single(i, w, x):
        """attention with kept first tokens, capped scores and a sink, or lightning attention"""
        q, k, v = (_mm(x, w[n]) for n in ("q", "k", "v"))
        out = torch.empty_like(q)
        for s, at in _spans(seqs):
            n = len(s.tokens)
            if i % 2 == 0:
                norm = lambda t, nw: _rms(t[at].reshape(n, -1, d), EPS) * w[nw].to(F64)  # noqa: E731
                out[at] = attention(i, s, norm(q, "q_norm"), norm(k, "k_norm"), v[at].reshape(n, kv, d), keep=4, cap=30.0, sink=w["sink"])
            else:
                head = lambda t: _silu(t[at]).reshape(n, sh // 2, 128)  # noqa: E731
                decay = torch.tensor(_decays(sh // 2), dtype=F64, device=DEV).expand(n, -1)
                out[at] = recurrence(i, s, head(q), head(k), head(v), decay).reshape(n, -1)
        if i % 2:
            out = _rms(out, EPS) * w["out_norm"].to(F64) * torch.sigmoid(_mm(x, w["g"]))
        return _mm(out, w["o"])

    for i in range(layers):
        w = _mixer_layer(case, i, seed)
        if not two:
            x = x + _rms(parallel(i, w, x), EPS) * w["norm1"].to(F64)
            x = x + _rms(_mm(_silu(_mm(x, w["gate"])) * _mm(x, w["up"]), w["down"]), EPS) * w["norm2"].to(F64)
            continue
        for j, f in (("1", lambda t: single(i, w, t)),
                     ("2", lambda t: _mm(torch.clamp(_mm(t, w["gate"]), min=0) * _mm(t, w["up"]), w["down"]))):
            into, out, mix = (w["hc%s_%s" % (j, n)].to(F64) for n in ("in", "out", "mix"))
            y = f(_rms((into[:, None, None] * xs).sum(0), EPS) * w["norm" + j].to(F64))
            xs = torch.einsum("st,snc->tnc", mix, xs) + out[:, None, None] * y
    xn = _rms(xs.sum(0) if two else x, EPS) * norm.to(F64)

    def logits(rows):
        lg = xn[rows] @ head.to(F64).t()
        return lg if two else 30.0 * torch.tanh(lg / 30.0)
    return logits


def exact(case, seed):
    """What `run` returns.  The greedy tokens are fed as the model is made to say them, all at once."""
    toks, op, new, batch = _tokens(case, seed), case["op"], case["new"], case["batch"]
    # a step of the tied model repeats its token
    step = 0 if case["model"] == "vekerax" else 1
    hist, ctx, seqs, rows, at = _history(case, seed), _contexts(case), [], [], 0
    first = None
    if op in ("generate", "prompt"):
        fed = toks[:case["tokens"]]
        if op == "generate":
            first = case["tokens"] - 1
            fed = fed + [fed[-1] + step * (j + 1) for j in range(new - 1)]
        seqs.append(_Sequence(fed, len(fed), 0, {}))
        rows = [len(fed) - 1]
    for b in range(batch if not seqs else 0):
        fed = [toks[b]] + _draft(case, toks[b]) if op == "verify" else [toks[b] + step * j for j in range(new)]
        keep = 3 if op == "verify" else new
        seqs.append(_Sequence(fed, keep, ctx[b], hist[b]))
        rows += list(range(at, at + len(fed))) if op == "verify" else [at + len(fed) - 1]
        at += len(fed)
    lg = (_hybrid64 if case["model"] == "hybrid" else _mixer64)(case, seed, seqs)
    logits = lg(rows)
    if op == "verify":
        tokens = logits.argmax(1).reshape(batch, DRAFT + 1)[:, :3]
    elif op == "generate":
        tokens = lg(list(range(first, first + new))).argmax(1)
    elif op == "prompt":
        tokens = logits.argmax(1)
    elif batch == 1:
        tokens = lg(list(range(new))).argmax(1)
    else:
        tokens = torch.stack([lg(list(range(a, batch * new, new))).argmax(1) for a in range(new)])
    if case["model"] == "hybrid":
        c = _hybrid_dims(case["size"])
        taps = [torch.stack(s.mem["new_taps"]) for s in seqs]
        conv = [_by_block(t, c["linear_num_key_heads"], c["linear_num_value_heads"], c["linear_key_head_dim"], c["linear_value_head_dim"]) for t in taps]
        return dict(tokens=tokens, logits=logits, S=torch.stack([torch.stack(s.mem["new_S"]) for s in seqs], 1), conv=torch.stack(conv, 1),
                    k=[torch.stack(s.mem["new_k"]) for s in seqs], v=[torch.stack(s.mem["new_v"]) for s in seqs])
    layers = SIZES[case["size"]][-1]
    i0, i1 = min(s.n0 for s in seqs), max(s.n0 + s.keep for s in seqs)

    def cache(name):
        out = []
        for i in range(layers):
            if name + str(i) not in {k[4:] for k in seqs[0].mem if k.startswith("new_")}:
                continue
            t = seqs[0].mem["new_" + name + str(i)]
            full = torch.zeros(len(seqs), i1, *t.shape[1:], dtype=F64, device=DEV)
            for b, s in enumerate(seqs):
                if s.n0:
                    full[b, :s.n0] = s.mem[name + str(i)].to(F64)
                full[b, s.n0:s.n0 + s.keep] = s.mem["new_" + name + str(i)]
            out.append(full[:, i0:])
        return out

    def states(name):
        return [torch.stack([s.mem["new_" + name + str(i)] for s in seqs]) for i in range(layers) if "new_" + name + str(i) in seqs[0].mem]
    return dict(tokens=tokens, logits=logits, S=states("S"), conv=states("conv"), k=cache("k"), v=cache("v"))
