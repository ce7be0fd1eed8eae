"""Prompts of many rows in one pass over the layers, and prompts that end a little behind a full pass, against short passes of the
same tokens: states per layer and head, caches per row, logits.  The passes cut the same chunks of the recurrences, so what
differs is the order of sums in the projections, rounded to the element type layer by layer."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(kind, max_seq, rows):
    from mi50grad_b200.config import EngineConfig, tiny_config, tiny_degedra_config, tiny_vekerax_config
    ecfg = EngineConfig(max_prompt_rows=rows)
    name, _, dtype = kind.partition(" ")
    if name == "hybrid":
        from mi50grad_b200.engine.engine import InferenceEngine
        from mi50grad_b200.models.weights import random_model
        eng = InferenceEngine(tiny_config(), max_seq_len=max_seq, engine_config=ecfg)
        eng.load_model(random_model(tiny_config(), 4))
        return eng
    if name == "degedra":
        from mi50grad_b200.engine.mixer_engine import MixerEngine
        eng = MixerEngine(tiny_degedra_config(), max_seq_len=max_seq, dtype=dtype, engine_config=ecfg)
    else:
        from mi50grad_b200.engine.vekerax_engine import VekeraxEngine
        eng = VekeraxEngine(tiny_vekerax_config(), max_seq_len=max_seq, dtype=dtype, engine_config=ecfg)
    eng.init_random(0)
    return eng


def _parts(eng, n):
    """(states [layer][head] flattened, cache rows [layer][row] flattened)"""
    st = eng.states
    if hasattr(st, "dn"):
        S, kv = [st.dn.S[i, 0] for i in range(st.dn.S.shape[0])], [t[i, 0, :n] for t in (st.kv.k, st.kv.v) for i in range(t.shape[0])]
    else:
        S, kv = [s[0] for s in st.S if s.numel()], [t[0, :n] for ts in (st.k, st.v) for t in ts if t.numel()]
    return [s.double().flatten(1) for s in S], [t.double().flatten(1) for t in kv]


def _worst(a, b, floor):
    """Largest relative 2-norm difference of a row of a and b; rows of less than `floor` of the mean norm count as that."""
    out = 0.0
    for x, y in zip(a, b):
        norm = y.norm(dim=1)
        out = max(out, float(((x - y).norm(dim=1) / norm.clamp_min(floor * norm.mean())).max()))
    return out


# 16-bit types: a value that rounds the other way moves a row by at most a step of its largest value or so, layer after
# layer (measured: no difference); 32 bits: sums of at most 320 products, over three to seven layers (measured 4e-5)
BOUND = {"hybrid": 4e-3, "degedra bfloat16": 2e-2, "degedra float32": 2e-4, "vekerax bfloat16": 2e-2, "vekerax float32": 2e-4}


@pytest.mark.parametrize("n", [1100, "pass + 61"])
@pytest.mark.parametrize("kind", BOUND)
def test_long_passes_equal_short_ones(kind, n):
    full = 4096 if kind == "hybrid" else 2048
    n = n if isinstance(n, int) else full + 61
    ids = torch.randint(0, 1000, (n,), generator=torch.Generator().manual_seed(9)).tolist()
    got = []
    for rows in (0, 512):
        eng = _engine(kind, n + 8, rows)
        eng.prefill_tokens(ids)
        assert eng.max_prefill == (rows or min(full, n + 8))
        got.append((*_parts(eng, n), eng.buf["logits"][:1].double()))
        eng.check_status()
    (S, kv, lg), (S2, kv2, lg2) = got
    assert len(S) and len(kv)
    assert _worst(S, S2, 0.1) < BOUND[kind] and _worst(kv, kv2, 0.1) < BOUND[kind]
    assert float((lg - lg2).norm() / lg2.norm()) < BOUND[kind]


@pytest.mark.parametrize("kind", ["degedra bfloat16", "vekerax bfloat16"])
def test_buffers_of_the_decode_step_come_before_those_of_prompts(kind):
    """The decode step's buffers do not lie between those of prompt passes, however long these are."""
    eng = _engine(kind, 3000, 0)
    eng._ensure_driver()
    names = list(eng.buf)
    decode = ["h", "xn", "proj", "attn_out", "act", "logits", "ss", "qbuf", "attn_scratch", "argmax_scratch", "rows", "row_tokens", "out_tokens"]
    assert max(names.index(n) for n in decode) < min(names.index(n) for n in ("p_h", "p_m", "p_xn", "p_proj", "p_attn", "p_act", "p_logits"))
