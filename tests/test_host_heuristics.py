"""Host-side choices that shape the GPU launches: the GEMV launch shape and the engine switches."""
import os

from mi50grad_b200.config import EngineConfig
from mi50grad_b200.ops.packing import GEMV_WK, launch_shape


def test_launch_shape_fills_one_wave_and_covers_k():
    for K, N in [(5120, 34816), (5120, 16384), (5120, 14336), (17408, 5120), (6144, 5120), (768, 5120), (2176, 5120),
                 (1536, 5120), (4352, 5120), (5120, 2048), (5120, 4352)]:
        KB, NTL = -(-K // 64), -(-N // 128) * 8
        ks, L = launch_shape(KB, NTL, 1)
        assert ks >= 1 and L >= 1
        assert ks * L * GEMV_WK >= KB                      # every k-block has an owner
        assert (ks - 1) * L * GEMV_WK < KB                 # no empty split
        assert (NTL * 16 // 128) * ks <= 2 * 148 or ks == 1   # two resident CTAs per SM, one wave
        # activation staging of one CTA stays inside its shared-memory share
        assert 2 * GEMV_WK * L * 2 * 64 <= 32_000


def test_launch_shape_short_k_is_not_split():
    # a row-parallel shard under 8-way tensor parallelism: the cross-CTA round trip costs more than it spreads
    for K in (768, 1024, 1536):
        ks, _ = launch_shape(-(-K // 64), 5120 // 16, 1)
        assert ks == 1


def test_launch_shape_more_rows_need_more_splits_or_shorter_slices():
    KB, NTL = 17408 // 64, 5120 // 16
    ks1, L1 = launch_shape(KB, NTL, 1)
    ks8, L8 = launch_shape(KB, NTL, 8)
    assert 2 * GEMV_WK * L8 * 9 * 64 <= 32_000
    assert ks8 >= ks1 and L8 <= L1


def test_engine_switch_defaults_and_environment(monkeypatch):
    for k in ("B200GRAD_CHAIN", "B200GRAD_SEQ_PARALLEL", "B200GRAD_AR_MODE", "B200GRAD_GRAPH", "B200GRAD_MULTIMEM"):
        monkeypatch.delenv(k, raising=False)
    e = EngineConfig()
    assert e.use_chain == -1 and e.seq_parallel == 1 and e.ar_mode == "exact" and e.use_graph and e.use_multimem
    monkeypatch.setenv("B200GRAD_CHAIN", "0")
    monkeypatch.setenv("B200GRAD_SEQ_PARALLEL", "0")
    e = EngineConfig()
    assert e.use_chain == 0 and e.seq_parallel == 0
    monkeypatch.setenv("B200GRAD_AR_MODE", "deferred_consistent")
    monkeypatch.setenv("B200GRAD_MULTIMEM", "0")
    e = EngineConfig.from_env()
    assert e.ar_mode == "deferred_consistent" and not e.use_multimem
    assert e.replace(use_chain=1).use_chain == 1 and e.use_chain == 0


def test_prompt_rows_and_their_memory():
    """A pass takes the rows it was given, never more than the default or the sequence; the budget knows its buffers."""
    import pytest
    from mi50grad_b200.config import PROMPT_ROWS, EngineConfig, memory_budget, prompt_rows, prompt_work_bytes, qwen35_27b
    assert prompt_rows(EngineConfig(), PROMPT_ROWS, 100000) == PROMPT_ROWS and prompt_rows(EngineConfig(), PROMPT_ROWS, 300) == 300
    assert prompt_rows(EngineConfig(max_prompt_rows=512), PROMPT_ROWS, 100000) == 512
    assert prompt_rows(EngineConfig(max_prompt_rows=9999), PROMPT_ROWS, 100000) == PROMPT_ROWS
    with pytest.raises(ValueError):
        EngineConfig(max_prompt_rows=8)
    cfg = qwen35_27b()
    work = prompt_work_bytes(cfg, 4096)
    assert 0.65e9 < work < 0.75e9 and work == 8 * prompt_work_bytes(cfg, 512)
    assert memory_budget(cfg, 4096)["scratch_gb"] >= work / 1e9



def test_fp16_gemv_slices_of_many_rows():
    """Five rows and more: slices of 4096 and longer become slices of 2560, none empty; up to four rows, and where slices are
    shorter, as the matrix was cut."""
    import ctypes as C
    from mi50grad_b200.ops import lib as L
    lib = L.lib()

    def shape(K, rows, ks, kslice):
        a, b = C.c_int(ks), C.c_int(kslice)
        lib.b2_gemv_f16_shape(K, rows, C.byref(a), C.byref(b))
        return a.value, b.value

    for K in list(range(256, 20000, 37)) + [2816, 3840, 4096, 5120, 8192, 17408, 65536]:
        cut = min(8192, -(-K // 256) * 256)
        given = (-(-K // cut), cut)
        assert shape(K, 4, *given) == given and shape(K, 8, -(-K // 3840), 3840) == (-(-K // 3840), 3840)
        for rows in (5, 8):
            ks, kslice = shape(K, rows, *given)
            assert (ks - 1) * kslice < K <= ks * kslice
            if cut < 4096:
                assert (ks, kslice) == given
            else:
                assert kslice == 2560
