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


def test_scan_splits_operands_with_rounding(K):
    """With orthogonal keys and no decay the matrix that a chunk's update starts from is beta on the diagonal, and the
    products that form it pass beta on as two TF32 terms.  What the terms leave out must not lean to one side: 512 errors of
    about 2^-24 at random are 3e-9 on the average; where the first term is cut off instead of rounded it is 7.5e-8."""
    import ctypes as C
    from mi50grad_b200.ops import lib as L
    dk, nv, T = 128, 16, 32
    cd = 2 * dk + nv * dk
    proj = torch.zeros(T, cd + nv * dk, device="cuda").half()
    proj[:, dk:dk + T] = torch.diag(torch.full((T,), 64.0, device="cuda")).half()      # keys: unit vectors
    proj[:, :dk] = 1.0
    proj[:, 2 * dk:cd] = 1.0
    ab = torch.randn(T, 2 * nv, generator=_gen(7), device="cuda").half()
    w = torch.zeros(cd, 4, device="cuda").half()
    w[:, 3] = 1.0
    conv, S = torch.zeros(1, nv, dk // 32, 2 * dk + 32, 3, device="cuda").half(), torch.zeros(1, nv, dk, dk, device="cuda")
    A, dtb, nw = torch.full((nv,), -100.0, device="cuda"), torch.zeros(nv, device="cuda").half(), torch.ones(dk, device="cuda").half()
    rows, seq_rows = K.make_rows([(0, 0, 0, 0, 1)] * T, "cuda"), torch.tensor([0, T], dtype=torch.int32, device="cuda")
    out, qk = torch.zeros(T, nv * dk, device="cuda").half(), torch.zeros(T, 2 * dk, device="cuda").half()
    L.lib().b2_deltanet_tw_floats.restype = C.c_longlong
    floats = int(L.lib().b2_deltanet_tw_floats(nv, T))
    tw = torch.zeros(floats, device="cuda")
    p = L.DeltaParams()
    p.proj, p.ld = proj.data_ptr(), proj.stride(0)
    p.off_q, p.off_k, p.off_v, p.off_z, p.off_a, p.off_b = 0, dk, 2 * dk, cd, -1, -1
    p.conv_w, p.conv_state, p.state = w.data_ptr(), conv.data_ptr(), S.data_ptr()
    p.A_log, p.dt_bias, p.norm_w = A.data_ptr(), dtb.data_ptr(), nw.data_ptr()
    p.seq_rows, p.rows, p.out, p.ldo = seq_rows.data_ptr(), rows.data_ptr(), out.data_ptr(), out.stride(0)
    p.nk, p.nv, p.n_seqs, p.eps, p.commit = 1, nv, 1, 1e-6, 0
    torch.cuda.synchronize()
    L.check(L.lib().b2_deltanet_chunk(C.byref(p), C.c_void_p(ab.data_ptr()), ab.stride(0), C.c_void_p(qk.data_ptr()), 2 * dk, T,
                                      C.c_void_p(tw.data_ptr()), dk, dk, L.stream()), "deltanet_chunk")
    wt = tw.view(nv, floats // nv)[:, :T * dk].view(nv, T, dk)                            # [head][row][key channel]
    beta = torch.sigmoid(ab[:, nv:].double()).t()
    got = torch.stack([wt[:, i, i] for i in range(T)], 1).double()
    assert abs(float((got / beta - 1).mean())) < 3e-8
