"""Which kernels a step of a matrix-state mixer launches, and what scratch memory it asks for: on the CPU, with the launches recorded."""
import pytest
import torch

from tessweave_engine_b200.csrc import ops
from tessweave_engine_b200.parts import PartSpec, Runtime, StateView, build_part
from tessweave_engine_b200.parts.base import StepContext, Workspace

HEADS, DIM = 4, 64
MODES = {"retention": ops.RECURRENCE_RETENTION, "mlstm": ops.RECURRENCE_MLSTM, "gated_delta": ops.RECURRENCE_DELTA}


def recur(kind, dtype, lens, monkeypatch, fixed=0):
    """(the launches as (name, most rows, below), the workspace's buffers) of a step of ``lens`` rows, or of ``fixed`` padding rows"""
    calls, rt = [], Runtime(torch.device("cpu"), dtype)
    monkeypatch.setattr(ops, "linear_recurrence", lambda *a, max_q_len, below, **k: calls.append(("tokens", max_q_len, below)))
    monkeypatch.setattr(ops, "recurrence_chunks", lambda *a, **k: calls.append(("chunks", a[15], ops.RECURRENCE_CHUNK_MIN_ROWS)))
    monkeypatch.setattr(ops, "load_library", lambda name, defines: calls.append(("load", name, defines["TW_DK"])))
    monkeypatch.setattr(ops, "delta_chunks", lambda *a, **k: calls.append(("chunks", a[12], ops.RECURRENCE_CHUNK_MIN_ROWS)))
    params = {"hidden": 32, "n_heads": HEADS, "key_dim": DIM, "value_dim": DIM, "eps": 1e-5}
    more = {"retention": {"decay": (0.9,) * HEADS}, "mlstm": {"gate_cap": 15.0}, "gated_delta": {"n_qk_heads": 2, "conv_taps": 4}}[kind]
    mixer = build_part("mixer", PartSpec(kind, {**params, **more}), rt)
    n = fixed or sum(lens)
    lens = [0] * min(n, 8) if fixed else lens
    i32 = torch.zeros(max(n, len(lens)), dtype=torch.int32)
    ctx = StepContext(runtime=rt, workspace=Workspace(rt.device), n_tokens=n, n_seqs=len(lens), token_ids=i32, positions=i32, seq_of_token=i32,
                      seq_slot=i32, seq_q_start=i32, seq_q_len=i32, seq_kv_len=i32, status=i32[:1], host_slot=lens, host_q_start=lens,
                      host_q_len=lens, host_kv_len=lens, max_q_len=1 if fixed else max(lens), max_kv_len=600, fixed_shape=bool(fixed))
    rows = torch.zeros(n, 3 * HEADS * DIM, dtype=torch.float32 if kind == "gated_delta" else dtype)
    q, k, v = (rows[:, i * HEADS * DIM:(i + 1) * HEADS * DIM] for i in range(3))
    extra = {"channel_decay": False, "qk_group": 2} if kind == "gated_delta" else {}
    mixer._recur(ctx, q, k, v, StateView(torch.zeros(1, mixer.state_numel)), True, **extra)
    return calls, {name: b.numel() for name, b in ctx.workspace._buffers.items() if "chunk" in name}


@pytest.mark.parametrize("kind", ["retention", "mlstm", "gated_delta"])
def test_float32_runs_go_token_by_token(kind, monkeypatch):
    calls, scratch = recur(kind, torch.float32, [700, 1, 64], monkeypatch)
    assert calls == [("tokens", 700, 0)] and not scratch
    assert recur(kind, torch.float32, [], monkeypatch, fixed=1000)[1] == {}


@pytest.mark.parametrize("kind", ["retention", "mlstm", "gated_delta"])
def test_requests_are_shared_out(kind, monkeypatch):
    """A long portion, and with it every request of enough rows, in chunks; the others by tokens; nobody twice and nobody left out."""
    enough, least = ops.recurrence_chunk_min_tokens(MODES[kind], DIM), ops.RECURRENCE_CHUNK_MIN_ROWS
    assert recur(kind, torch.bfloat16, [enough, least, least - 1, 1], monkeypatch)[0] == [("chunks", enough, least), ("tokens", least - 1, least)]
    assert recur(kind, torch.bfloat16, [enough, least], monkeypatch)[0] == [("chunks", enough, least)]
    assert recur(kind, torch.bfloat16, [enough - 1, least, 1], monkeypatch)[0] == [("tokens", enough - 1, 0)]


@pytest.mark.parametrize("kind", ["retention", "mlstm", "gated_delta"])
def test_scratch_is_asked_for_where_a_portion_can_be_long_enough(kind, monkeypatch):
    """A padding step, whose buffers a workspace keeps, asks for no more chunks than a step of its size can be cut into, and for none
    where the step has no room for a portion that goes in chunks; what a step needs is never more than what it asked for."""
    enough = ops.recurrence_chunk_min_tokens(MODES[kind], DIM)
    main = "recurrence.delta_chunks" if kind == "gated_delta" else "recurrence.chunk_state"
    per_chunk = ops.delta_chunk_floats(HEADS, 2, DIM, DIM) if kind == "gated_delta" else HEADS * DIM * (DIM + 1)
    for n in (1, 8, 64, 256, enough - 1):
        calls, scratch = recur(kind, torch.bfloat16, [], monkeypatch, fixed=n)
        assert calls == [("tokens", 1, 0)] and not scratch
    library = ("load", "delta_chunks" if kind == "gated_delta" else "recurrence_chunks", DIM)
    for n in (enough, 2112):
        calls, held = recur(kind, torch.bfloat16, [], monkeypatch, fixed=n)
        # (the library is loaded, and where need be built, before the first prompt waits for it)
        assert calls == [library, ("tokens", 1, 0)] and held[main] == ops.recurrence_chunk_count(n, 8) * per_chunk
        for lens in ([n], [enough] + [32] * min(7, (n - enough) // 32), [n - 7] + [1] * 7 if n > enough + 7 else [n]):
            _, used = recur(kind, torch.bfloat16, lens, monkeypatch)
            assert used.keys() == held.keys() and all(used[name] <= held[name] for name in used)


def test_every_key_size_of_the_chunks_has_its_line():
    for mode, line in ((ops.RECURRENCE_RETENTION, ops.RECURRENCE_CHUNK_MIN_TOKENS), (ops.RECURRENCE_MLSTM, ops.RECURRENCE_CHUNK_MIN_TOKENS)):
        assert sorted(line) == [d for d in range(1, 257) if ops.recurrence_chunks_supported(mode, torch.bfloat16, d, 64)]
    rows = torch.zeros(4, 256)
    assert sorted(ops.DELTA_CHUNK_MIN_TOKENS) == [d for d in range(1, 257) if ops.delta_chunks_supported(rows, rows, d, 64, False)]
    assert min(min(ops.RECURRENCE_CHUNK_MIN_TOKENS.values()), min(ops.DELTA_CHUNK_MIN_TOKENS.values())) >= ops.RECURRENCE_CHUNK_MIN_ROWS


def test_every_key_size_of_the_chunks_is_built_ahead():
    from tessweave_engine_b200.csrc.variants import default_variants
    for name, mode in (("recurrence_chunks", ops.RECURRENCE_RETENTION), ("recurrence_chunks", ops.RECURRENCE_MLSTM)):
        sizes = [d for d in range(1, 257) if ops.recurrence_chunks_supported(mode, torch.bfloat16, d, 64)]
        assert [v["TW_DK"] for v in default_variants(name)] == sizes
    rows = torch.zeros(4, 256)
    sizes = [d for d in range(1, 257) if ops.delta_chunks_supported(rows, rows, d, 64, False)]
    assert [v["TW_DK"] for v in default_variants("delta_chunks")] == sizes


@pytest.mark.parametrize("key_dim", [64, 128])
@pytest.mark.parametrize("heads,value_dim", [(14, 128), (14, 64), (8, 128), (6, 64), (32, 128)])
def test_width_of_the_delta_rules_walk(key_dim, heads, value_dim):
    """A block of the walk takes 32 values only where the step's last block ends earlier so, laid out block by block over the SMs; in
    particular never where blocks of 16 values all run at once, whatever else the step brings."""
    def ends(lens, values):
        free = [0.0] * 148
        for m in sorted(lens, reverse=True) if len(lens) <= 32 else lens:
            for _ in range(heads * value_dim // values if m >= ops.RECURRENCE_CHUNK_MIN_ROWS else 0):
                at = free.index(min(free))
                free[at] += ops.DELTA_WALK_START_US + ops.DELTA_WALK_CHUNK_US[key_dim][values // 32] * -(-m // 64)
        return max(free)

    for lens in ([2048], [2048, 1], [2048] + [1] * 30, [1] * 40 + [2048], [777, 1024, 201], [1900, 60, 80], [1500, 300], [1200, 400, 200], [1000, 1000],
                 [31, 600, 600, 600], [512] * 4, [64] * 20 + [800], [800] + [33] * 40, [1024] * 8):
        narrow, wide = ends(lens, 16), ends(lens, 32)
        taken = ops.delta_walk_values(lens, heads, key_dim, value_dim)
        assert abs(ends(lens, taken) - min(narrow, wide)) < 1e-6, lens
        if sum(m >= ops.RECURRENCE_CHUNK_MIN_ROWS for m in lens) * heads * value_dim // 16 <= 148:
            assert taken == 16


def test_a_step_says_how_wide_its_walk_is(monkeypatch):
    """(14 heads of 128 x 128 would take 32 values for the portions; the heads of the mixer here and its one long portion take 16)"""
    assert ops.delta_walk_values([777, 1024, 201], 14, 128, 128) == 32 and ops.delta_walk_values([2048] + [1] * 30, 14, 128, 128) == 16
    seen = []
    with monkeypatch.context() as m:
        m.setattr(ops, "delta_walk_values", lambda lens, *sizes: seen.append((lens, *sizes)) or 16)
        recur("gated_delta", torch.bfloat16, [700, 1, 64], m)
    assert seen == [([700, 1, 64], HEADS, DIM, DIM)]
