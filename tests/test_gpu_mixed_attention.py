"""Steps of prompt portions and single tokens: the two attention kernels side by side, over the row tiles there are."""
import pytest
import torch

from test_gpu_kernels import dense_attention, dev, ops, paged_setup, status


@pytest.mark.gpu
@pytest.mark.parametrize("hq,hkv,d,window", [(28, 4, 128, 0), (8, 8, 64, 0), (10, 2, 128, 70)])
@pytest.mark.parametrize("order", ["portions first", "portions last", "portion at 31, 32 and 40"])
def test_prompt_and_decode_attention_side_by_side(hq, hkv, d, window, order):
    """Row tiles found through the requests' row counts (more than a warp's 32 requests, portions at both sides of the 32nd, of one
    row tile and of several, a step's first and last request) give the bits of the grid that has every request's most tiles, and
    the decode attention that runs beside gives the bits of the one that waits.  Both against plain attention."""
    o, n = ops(), 43
    at = {"portions first": (0, 1, 2), "portions last": (40, 41, 42), "portion at 31, 32 and 40": (31, 32, 40)}[order]
    rows = [1] * n
    for i, m in zip(at, (37, 300, 2)):
        rows[i] = m
    held = [(i * 37) % 230 for i in range(n)]
    total = [a + b for a, b in zip(rows, held)]
    setup = paged_setup(total, 16, hkv, d, torch.bfloat16, seed=hq)
    starts = [sum(rows[:i]) for i in range(n)]
    q = dev(torch.randn(sum(rows), hq * d, generator=torch.Generator().manual_seed(4)), torch.bfloat16)
    i32 = lambda v: dev(torch.tensor(v, dtype=torch.int32))     # noqa: E731
    meta = (i32(starts), i32(rows), i32(total), i32(setup["slots"]), setup["table"], setup["k_pages"], setup["v_pages"], n)
    nsplit = 2
    scratch = torch.zeros(o.decode_scratch_floats(hq, d), device="cuda")
    counters = torch.zeros(o.decode_counter_ints(n, hkv, hq // hkv), dtype=torch.int32, device="cuda")
    results = []
    for counted, beside in ((False, False), (True, False), (True, True), (False, True)):
        for _ in range(3):      # (several times: the kernels' blocks meet in another order each time)
            out, st = torch.full((sum(rows), hq * d), 7.0, dtype=torch.bfloat16, device="cuda"), status()
            q2 = q + 0          # (what the kernel before the prompts' leaves is what both read)
            o.attention_prefill_tcgen05(out, q2, *meta, max(rows), hq, hkv, d, window, d ** -0.5, True, st,
                                        host_q_len=rows if counted else None)
            o.attention_decode_tma(out, q2, None, None, None, False, *meta, hq, hkv, d, window, d ** -0.5, nsplit, scratch, counters, st,
                                   beside_prompts=beside)
            results.append(out + 0)
            assert int(st.cpu()[0]) == 0
    assert all(torch.equal(results[0], r) for r in results[1:])
    got = results[0].float().cpu().view(-1, hq, d)
    for i in sorted({*at, 0, 7, 42}):
        pos = list(range(held[i], total[i]))
        want = dense_attention(q.float().cpu().view(-1, hq, d)[starts[i]:starts[i] + rows[i]], setup["k"][i].bfloat16().float(),
                               setup["v"][i].bfloat16().float(), pos, window or None)
        assert torch.allclose(got[starts[i]:starts[i] + rows[i]], want, rtol=2e-2, atol=2e-2), f"request {i}"


@pytest.mark.gpu
@pytest.mark.parametrize("captured", [False, True])
def test_what_the_kernel_before_both_wrote_is_seen(captured):
    """The queries, and every request's newest keys and values, written into fresh pages by the kernel right before the prompts'
    attention: the decode attention beside it (the word between the two set) gives the bits of the one that waits, plainly and in a
    graph, and the word is zero again."""
    o, hq, hkv, d, rows = ops(), 28, 4, 128, [300, 1, 1, 260] + [1] * 28
    n, held = len(rows), [(i * 53) % 900 for i in range(len(rows))]
    total = [a + b for a, b in zip(rows, held)]
    g = torch.Generator().manual_seed(9)
    setup = paged_setup(total, 16, hkv, d, torch.bfloat16, seed=3)
    starts = [sum(rows[:i]) for i in range(n)]
    i32 = lambda v: dev(torch.tensor(v, dtype=torch.int32))     # noqa: E731
    meta = (i32(starts), i32(rows), i32(total), i32(setup["slots"]), setup["table"], setup["k_pages"], setup["v_pages"], n)
    positions = i32([p for i in range(n) for p in range(held[i], total[i])])
    seq = i32([i for i in range(n) for _ in range(rows[i])])
    scratch = torch.zeros(o.decode_scratch_floats(hq, d), device="cuda")
    counters = torch.zeros(o.decode_counter_ints(n, hkv, hq // hkv), dtype=torch.int32, device="cuda")
    ready = torch.zeros(1, dtype=torch.int32, device="cuda")
    made = dev(torch.randn(2, sum(rows), (hq + 2 * hkv) * d, generator=g), torch.bfloat16)     # two steps' products
    inv_freq = dev((1e4 ** (-torch.arange(0, d, 2) / d)).float())
    st = status()

    def step(which, word):
        out, qkv = torch.zeros(sum(rows), hq * d, dtype=torch.bfloat16, device="cuda"), made[which] + 0
        o.rope_kv_write(qkv, None, positions, seq, meta[3], setup["table"], inv_freq, setup["k_pages"], setup["v_pages"], sum(rows), hq, hkv,
                        d, True, st)
        q = qkv[:, :hq * d]
        o.attention_prefill_tcgen05(out, q, *meta, max(rows), hq, hkv, d, 0, d ** -0.5, True, st, host_q_len=rows, ready=word)
        o.attention_decode_tma(out, q, None, None, None, False, *meta, hq, hkv, d, 0, d ** -0.5, 2, scratch, counters, st,
                               beside_prompts=word is not None, ready=word)
        return out

    def both(word):
        for _ in range(3):
            outs = [step(0, word), step(1, word)]       # (the second step writes over the first one's keys and values)
        return [t + 0 for t in outs]

    want = both(None)
    if captured:
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            both(ready)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = both(ready)
        for _ in range(3):
            graph.replay()
    else:
        got = both(ready)
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and not torch.equal(want[0], want[1])
    assert int(ready) == 0 and int(st) == 0


@pytest.mark.gpu
def test_behind_anything_else_it_waits():
    """A decode attention whose word nobody set waits for the kernel before it, here one that lets it start long before its own
    results, the queries, are written."""
    o, hq, hkv, d, n, k = ops(), 28, 4, 128, 40, 8192
    g = torch.Generator().manual_seed(5)
    total = [1 + (i * 37) % 300 for i in range(n)]
    setup = paged_setup(total, 16, hkv, d, torch.bfloat16, seed=2)
    i32 = lambda v: dev(torch.tensor(v, dtype=torch.int32))     # noqa: E731
    meta = (i32(range(n)), i32([1] * n), i32(total), i32(setup["slots"]), setup["table"], setup["k_pages"], setup["v_pages"], n)
    scratch = torch.zeros(o.decode_scratch_floats(hq, d), device="cuda")
    counters = torch.zeros(o.decode_counter_ints(n, hkv, hq // hkv), dtype=torch.int32, device="cuda")
    ready, st = torch.zeros(1, dtype=torch.int32, device="cuda"), status()
    x, w = dev(torch.randn(n, k, generator=g), torch.bfloat16), dev(torch.randn(hq * d, k, generator=g) / 90, torch.bfloat16)

    def run(beside):
        q, out = torch.full((n, hq * d), 3.0, dtype=torch.bfloat16, device="cuda"), torch.zeros(n, hq * d, dtype=torch.bfloat16, device="cuda")
        o.gemm_small_m(q, x, w, n, early_dependents=True)
        o.attention_decode_tma(out, q, None, None, None, False, *meta, hq, hkv, d, 0, d ** -0.5, 2, scratch, counters, st, beside_prompts=beside,
                               ready=ready)
        return out

    want = run(False)
    assert all(torch.equal(run(True), want) for _ in range(5)) and int(ready) == 0 and int(st) == 0


@pytest.mark.gpu
def test_only_a_decode_attention_with_q_given_runs_beside():
    o = ops()
    setup = paged_setup([40], 16, 1, 64, torch.bfloat16)
    i32 = lambda v: dev(torch.tensor(v, dtype=torch.int32))     # noqa: E731
    qkv = dev(torch.randn(1, 3 * 64), torch.bfloat16)
    with pytest.raises(Exception, match="beside"):
        o.attention_decode_tma(torch.empty(1, 64, dtype=torch.bfloat16, device="cuda"), None, qkv, None, None, False, i32([0]), i32([1]),
                               i32([40]), i32(setup["slots"]), setup["table"], setup["k_pages"], setup["v_pages"], 1, 1, 1, 64, 0, 0.125,
                               1, None, None, status(), beside_prompts=True)
