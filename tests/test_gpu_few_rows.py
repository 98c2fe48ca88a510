"""Kernels of decode steps that run a row's chain in parallel, against the kernels of many rows."""
import pytest
import torch


def ops():
    from tessweave_engine_b200.csrc import ops as o
    return o


@pytest.mark.gpu
@pytest.mark.parametrize("ranks,rot,gates", [((1536, 192), 64, 28), ((128, 8), 0, 0), ((2048, 264), 32, 40), ((136, 512), 72, 5)])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("own_rows,write_cache", [(True, True), (False, False)])
def test_rows_of_attention_over_latents(ranks, rot, gates, interleaved, own_rows, write_cache):
    """Up to 64 rows (a warp or more for each span, the rotation and the gates) give the bits of steps with more: the norms, the rotated
    part, the cached rows and the gates; a row of no request is left alone, a page that is not there is reported."""
    o, few, many, page = ops(), 9, 70, 16
    g = torch.Generator().manual_seed(sum(ranks) + rot)
    q_rank, kv_rank = ranks
    head = kv_rank + rot
    width = -(-(q_rank + head + gates) // 8) * 8
    rows = torch.randn(many, width, generator=g).bfloat16().cuda()
    seq = torch.arange(many, dtype=torch.int32)
    seq[few - 2] = -1
    i32 = lambda t: t.to(torch.int32).cuda()        # noqa: E731
    positions, slots = torch.randint(0, 5 * page, (many,), generator=g), torch.randperm(many, generator=g)
    table = torch.arange(many * 5).view(many, 5)
    table[slots[1]] = -1                            # request 1 holds no page
    w0, w1 = torch.randn(q_rank, generator=g).cuda(), torch.randn(kv_rank, generator=g).cuda()
    inv_freq = (10000.0 ** (-torch.arange(0, max(rot, 2), 2) / max(rot, 2))).float().cuda()

    def run(n):
        x = rows[:n].clone()
        cache = torch.full((many * 5, 1, page, head), 9.0, dtype=torch.bfloat16, device="cuda")
        first = torch.full((n, q_rank), 5.0, dtype=torch.bfloat16, device="cuda") if own_rows else None
        gate = torch.full((n, gates), 5.0, device="cuda") if gates else None
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        o.norm_rotate_store(x, n, [(0, 1, q_rank, w0), (q_rank, 1, kv_rank, w1)], 1e-6, i32(positions[:n]), i32(seq[:n]), i32(slots), i32(table),
                            cache, None, q_rank, q_rank, write_cache, status, dst0=first, rot_col=q_rank + kv_rank, rot_dims=rot,
                            inv_freq=inv_freq if rot else None, interleaved=interleaved, magnitude=1.1, gate_col=q_rank + head, gate_out=gate)
        held = cache[table.clamp_min(0)[slots[:few]].cuda()]       # the pages of the few rows' requests
        return x[:few], None if first is None else first[:few], None if gate is None else gate[:few], held, int(status) if write_cache else 0

    got, want = run(few), run(many)
    for a, b in zip(got, want):
        assert a == b if isinstance(a, int) else a is None and b is None or torch.equal(a, b)
    assert got[4] == (2 if write_cache else 0)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,width,experts,stride", [(1, 8, 2, 8), (8, 3584, 8, 3584), (148, 1032, 5, 1040), (33, 264, 64, 264)])
@pytest.mark.parametrize("shared,scored", [(True, False), (False, True)])
def test_router_reads_rows_where_they_lie(rows, width, experts, stride, shared, scored):
    """Few bf16 rows on 16-byte boundaries are routed without staging them, and beside a product: the bits of rows that are staged
    (here: rows that start off a boundary)."""
    o = ops()
    g = torch.Generator().manual_seed(rows + width)
    top, dev = min(2, experts), "cuda"
    h = torch.randn(rows, width, generator=g).bfloat16()
    wr, ws = torch.randn(experts, width, generator=g).bfloat16().to(dev), torch.randn(width, generator=g).bfloat16().to(dev)
    br = torch.randn(experts, generator=g).to(dev)
    weights = torch.randn(64, width, generator=g).bfloat16().to(dev)

    ready = torch.zeros(1, dtype=torch.int32, device=dev)

    def run(x, beside):
        chosen, weight = torch.empty(rows, top, dtype=torch.int32, device=dev), torch.empty(rows, top, device=dev)
        gate = torch.empty(rows, device=dev) if shared else None
        if beside:
            out = torch.empty(rows, 64, dtype=torch.bfloat16, device=dev)
            if beside == "rows made just before":
                x = x + 0
            o.gemm_small_m(out, x, weights, rows, early_dependents=True, ready=ready)
        o.moe_route(chosen, weight, gate, x, wr, br, ws if shared else None, rows, top, score_all=scored, beside=bool(beside), ready=ready)
        return [t for t in (chosen, weight, gate) if t is not None] + ([out] if beside else [])

    def laid(offset, row):
        x = torch.zeros(rows * row + 8, dtype=torch.bfloat16, device=dev)[offset:offset + rows * row].view(rows, row)[:, :width]
        x.copy_(h)
        return x

    want = run(laid(1, stride + 1), False)
    assert all(torch.equal(a, b) for a, b in zip(run(laid(0, stride), False), want))
    if rows <= 64 and stride == width:
        for i in range(4):
            got = run(laid(0, stride), "rows made just before" if i & 1 else True)
            assert int(ready) == 0
            assert all(torch.equal(a, b) for a, b in zip(got, want))
            assert torch.allclose(got[-1].float(), (h.to(dev).float() @ weights.float().T), rtol=2e-2, atol=2e-2 * width ** 0.5)


@pytest.mark.gpu
def test_router_behind_anything_else_waits():
    """A router whose word nobody set waits for the kernel before it, here one that lets it start long before its own results, the
    router's rows, are written; a product without a kernel beside it takes no word."""
    o, rows, width, k = ops(), 40, 3584, 8192
    g = torch.Generator().manual_seed(8)
    make = lambda *shape: torch.randn(*shape, generator=g).bfloat16().cuda()        # noqa: E731
    x, w, wr, ready = make(rows, k), make(width, k) / 90, make(8, width), torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(beside):
        h = torch.full((rows, width), 3.0, dtype=torch.bfloat16, device="cuda")
        chosen, weight = torch.empty(rows, 2, dtype=torch.int32, device="cuda"), torch.empty(rows, 2, device="cuda")
        o.gemm_small_m(h, x, w, rows, early_dependents=True)
        o.moe_route(chosen, weight, None, h, wr, None, None, rows, 2, beside=beside, ready=ready)
        return chosen, weight

    want = run(False)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(run(True), want)) and int(ready) == 0
    with pytest.raises(Exception, match="beside"):
        o.gemm_small_m(torch.empty(rows, width, dtype=torch.bfloat16, device="cuda"), x, w, rows, ready=ready)
