"""Kernels that sum on the tensor cores or split their operands, against 64 bits: what is computed in 32 bits stays so.

The tensor core cuts off the bits below its 24 at every addition, so long chains of its sums drift towards zero, which a
tolerance in 16-bit steps does not show.  Here 16-bit results are compared with the correctly rounded ones (an error of e
relative moves one over the border with a probability of about 2 e / 2^-11), 32-bit ones directly."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from mi50grad_b200.ops import kernels
    return kernels


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _attention(q, k, v, nq, nkv, mask=None):
    """64-bit attention of rows of one sequence."""
    hd = k.shape[-1]
    s = torch.einsum("rkgd,tkd->rkgt", q.double().view(-1, nkv, nq // nkv, hd), k.double()) * hd ** -0.5
    if mask is not None:
        s = s.masked_fill(~mask[:, None, None], -float("inf"))
    return torch.einsum("rkgt,tkd->rkgd", torch.softmax(s, -1), v.double()).reshape(-1, nq * hd)


def _misrounded(out, ref):
    return float((out.double() != ref.half().double()).double().mean())


@pytest.mark.parametrize("hd,splits", [(256, 8), (128, 32), (64, 8)])
def test_decode_attention_weights_far_below_the_maximum(K, hd, splits):
    """60000 slots of e^-19 of the largest weight each: alone none is 2^-27 of it, together they are the result, because
    the value of the heaviest slot is zero."""
    n = 60000
    q = torch.zeros(1, 2 * hd, device="cuda").half()
    q[:, ::hd] = 8.0
    k, v = torch.zeros(1, n + 1, 1, hd, device="cuda").half(), torch.ones(1, n + 1, 1, hd, device="cuda").half()
    k[0, 777, 0, 0] = 19.0 * hd ** 0.5 / 8.0
    v[0, 777] = 0.0
    out = K.decode_attn(q, K.make_rows([(0, n, n, n, 1)], "cuda"), k, v, 2, 1, hd, splits=splits)
    ref = _attention(q, k[0], v[0], 2, 1)
    assert float(((out.double() - ref) / ref).abs().max()) < 1e-3       # one rounding to fp16, 2^-11


@pytest.mark.parametrize("hd,nq,nkv,ctx,splits", [(256, 6, 1, 8000, 4), (128, 8, 2, 3000, 1), (64, 8, 1, 5000, 2)])
def test_decode_attention_sums_round(K, hd, nq, nkv, ctx, splits):
    """Values that lean to one side, so that sums that are cut off show: at most a few roundings of 2^-24."""
    g = _gen(3)
    q = torch.randn(6, nq * hd, generator=g, device="cuda").half()
    k = torch.randn(1, ctx + 1, nkv, hd, generator=g, device="cuda").half()
    v = (torch.randn(1, ctx + 1, nkv, hd, generator=g, device="cuda") * 2 + 3).half()
    out = K.decode_attn(q, K.make_rows([(0, ctx, ctx, ctx, 1)] * 6, "cuda"), k, v, nq, nkv, hd, splits=splits)
    assert _misrounded(out, _attention(q, k[0], v[0], nq, nkv)) < 1.5e-3


@pytest.mark.parametrize("N,Kd,rows", [(1000, 5120, 5), (1024, 17408, 8), (512, 2048, 2)])
def test_gemv_f16_of_several_rows_sums_round(K, N, Kd, rows):
    """A sum of K products in fp32: a rounding of 2^-24 for each of the about 100 additions of an output's longest chain,
    of random sign, is 1.5e-7 at most; one that is cut off every time loses several times that."""
    from mi50grad_b200.engine.engine import DeviceLinear
    from mi50grad_b200.ops import lib as L
    g = _gen(4)
    for positive in (False, True):
        w, x = torch.randn(N, Kd, generator=g, device="cuda") * 0.02, torch.randn(rows, Kd, generator=g, device="cuda")
        w, x = (w.abs().half(), x.abs().half()) if positive else (w.half(), x.half())
        out = torch.zeros(rows, N, device="cuda")
        K.gemv(DeviceLinear(dense=w), x, out=out, mode=L.EPI_STORE_F32)
        ref = x.double() @ w.double().t()
        assert float((out.double() - ref).norm() / ref.norm()) < 2e-7


def test_gate_projections_sums_round(K):
    g = _gen(5)
    x, wa, wb = (torch.randn(n, 5120, generator=g, device="cuda").half() for n in (160, 48, 48))
    out = K.ab_proj(x, wa, wb)[:, :96]
    assert _misrounded(out, torch.cat([x.double() @ wa.double().t(), x.double() @ wb.double().t()], 1)) < 1.5e-3


@pytest.mark.parametrize("hd,T,past", [(256, 300, 1200), (64, 300, 1200)])
def test_prompt_attention_with_peaked_scores(K, hd, T, past):
    """Where one weight outweighs the others, it is exactly 1 in fp16 and the result little more than its rounding to
    fp16 (2.1e-4 in the 2-norm) away."""
    g = _gen(6)
    n = past + T
    q = (torch.randn(T, 2 * hd, generator=g, device="cuda") * 2.5).half()
    k = torch.randn(1, n, 1, hd, generator=g, device="cuda").half()
    v = (torch.randn(1, n, 1, hd, generator=g, device="cuda") * 2).half()
    out = K.attn_prefill_tc(q, K.make_rows([(0, past + i, past + i, past + i + 1, 0) for i in range(T)], "cuda"), k, v, 2, 1, hd)
    K.gemm_tc_check_status()
    mask = torch.arange(n, device="cuda")[None] <= past + torch.arange(T, device="cuda")[:, None]
    ref = _attention(q, k[0], v[0], 2, 1, mask)
    assert float((out.double() - ref).norm() / ref.norm()) < 2.4e-4
