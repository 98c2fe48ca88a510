"""The walk of the gated delta rule's chunks with many requests: 16 or 32 values a block, the longest request first."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("heads,dk,dv,lens", [(2, 64, 64, [33, 64, 65, 64, 7, 129] * 6), (2, 128, 128, [64, 200, 64, 31, 130] * 5),
                                              (4, 64, 128, [65, 65, 65, 190, 32, 65])])
@pytest.mark.parametrize("values", [16, 32])
def test_requests_together_and_alone(heads, dk, dv, lens, values):
    """A step whose blocks take 16 or 32 values (more than a warp's 32 requests, requests of one length, short ones left to the token
    kernel) gives the bits of every request alone, whose blocks take 16."""
    from tessweave_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(heads * dk)
    n, half, count = sum(lens), heads // 2, len(lens)
    assert dv // 16 * heads * count > 148 >= dv // 16 * heads
    unit = lambda: torch.nn.functional.normalize(torch.randn(n, half, dk, generator=g), dim=-1).view(n, -1).cuda()       # noqa: E731
    q, k, v = unit(), unit(), torch.randn(n, heads * dv, generator=g).cuda()
    pre, write = torch.randn(n, heads, generator=g).cuda(), torch.randn(n, heads, generator=g).cuda()
    args = {"p0": torch.linspace(-5, 0, heads).cuda(), "p1": torch.randn(heads, generator=g).cuda(), "qk_group": 2}
    state = torch.randn(count, heads * dk * dv, generator=g).cuda()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")          # noqa: E731
    starts = [sum(lens[:i]) for i in range(count)]
    slots = torch.randperm(count, generator=g).tolist()

    def run(st, which, values=16):
        rows = slice(starts[which[0]], starts[which[-1]] + lens[which[-1]])
        m = rows.stop - rows.start
        out = torch.full((m, heads * dv), -7.0, device="cuda")
        chunks = ops.recurrence_chunk_count(m, len(which))
        scratch = torch.full((chunks * ops.delta_chunk_floats(heads, 2, dk, dv),), float("nan"), device="cuda")
        ops.delta_chunks(out, q[rows], k[rows], v[rows], st, i32([slots[i] for i in which]), i32([starts[i] - rows.start for i in which]),
                         i32([lens[i] for i in which]), len(which), heads, dk, dv, max(lens[i] for i in which), scratch, True,
                         pre=pre[rows], write_pre=write[rows], walk_values=values, **args)
        return out

    together, alone = state.clone(), state.clone()
    got = run(together, list(range(count)), values)
    left = lambda m: torch.full((m, heads * dv), -7.0, device="cuda")          # noqa: E731
    want = torch.cat([run(alone, [i]) if m >= 32 else left(m) for i, m in enumerate(lens)])
    assert torch.equal(got, want) and torch.equal(together, alone)
