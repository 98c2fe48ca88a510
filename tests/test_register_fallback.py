"""Kernels whose roles split a block's registers, compiled with another count: what they would serve goes another way."""
from types import SimpleNamespace

import pytest
import torch

from tessweave_engine_b200.csrc import ops
from tessweave_engine_b200.parts.attention import PagedSoftmaxMixer


class FakeLibrary:
    def __init__(self, answer):
        self.answers, self.asked = list(answer), 0

    def __getattr__(self, name):
        def ask():
            self.asked += 1
            return self.answers.pop(0)
        return ask


@pytest.mark.parametrize("answers,want,asked", [([1], [True, True], 1), ([0], [False, False], 1), ([-3, 1], [True, True], 2), ([-3, 0], [True, False], 2)])
def test_a_library_is_asked_once_and_a_failed_question_is_not_kept(answers, want, asked, monkeypatch):
    lib = FakeLibrary(answers)
    monkeypatch.setattr(ops, "load_library", lambda name, defines=None: lib)
    monkeypatch.setattr(ops, "_built", {})
    assert [ops.gemm_fp32_built() for _ in want] == want and lib.asked == asked


@pytest.mark.parametrize("built", [True, False])
def test_prompt_attention_falls_back_to_the_register_kernel(built, monkeypatch):
    calls = []
    for name in ("attention_prefill", "attention_prefill_tcgen05"):
        monkeypatch.setattr(ops, name, lambda *a, _name=name, **k: calls.append(_name))
    monkeypatch.setattr(ops, "tcgen05_attention_built", lambda head_dim, v_dim: built)
    mixer = SimpleNamespace(score_terms=False, scale=0.1, runtime=SimpleNamespace(dtype=torch.bfloat16), head_dim=128, v_dim=128, n_heads=4,
                            n_kv_heads=2, reach=0, _prefill_own=lambda *a: False, _terms=dict)
    cache = SimpleNamespace(k_pages=torch.zeros(1, 2, 16, 128), v_pages=None, block_table=None)
    ctx = SimpleNamespace(decode_only=False, fixed_shape=False, host_q_len=[300], max_q_len=300, n_seqs=1, seq_q_start=None, seq_q_len=None,
                          seq_kv_len=None, seq_slot=None, status=None)
    PagedSoftmaxMixer._attend_tensor_cores(mixer, ctx, None, None, cache)
    assert calls == ["attention_prefill_tcgen05" if built else "attention_prefill"]


@pytest.mark.gpu
def test_kernels_as_built_here_can_run_and_a_product_goes_to_the_library_where_one_cannot(monkeypatch):
    from tessweave_engine_b200.parts.base import Workspace
    from tessweave_engine_b200.parts.linear import linear
    assert ops.gemm_fp32_built()
    assert all(ops.tcgen05_attention_built(d, v) for d in (64, 128) for v in (32, 64, 128))
    x, w = torch.randn(800, 256, device="cuda"), torch.randn(1024, 256, device="cuda")
    ctx = SimpleNamespace(workspace=Workspace(torch.device("cuda")), status=torch.zeros(1, dtype=torch.int32, device="cuda"))
    want, calls = x.double() @ w.double().T, []
    monkeypatch.setattr(ops, "CALL_LOG", calls)
    for built in (True, False):
        monkeypatch.setattr(ops, "gemm_fp32_built", lambda built=built: built)
        got = linear(ctx, "y", x, w)
        assert float((got.double() - want).norm() / want.norm()) < 1e-6 and ("tw_gemm_fp32" in calls) == built
        calls.clear()
