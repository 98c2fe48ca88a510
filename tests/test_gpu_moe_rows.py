"""Routed experts: the products of steps with few rows, the router's two kernels, the passes over sorted rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def sorted_pairs(ops, chosen, experts):
    n, top = chosen.shape
    i32 = lambda k: torch.full((k,), -7, dtype=torch.int32, device="cuda")         # noqa: E731
    order, place, ends = i32(n * top), i32(n * top), i32(experts)
    ops.moe_sort(order, place, ends, chosen, n)
    return order, place, ends


@pytest.mark.parametrize("rows,width,experts,shared,how", [(128, 64, 3, False, 0), (130, 1160, 8, True, 0), (129, 3584, 20, True, 1),
                                                           (200, 776, 12, False, 2)])
def test_router_of_many_rows(rows, width, experts, shared, how):
    """The kernel for steps of many rows chooses and weighs, bit for bit, as the one for few."""
    from tessweave_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(width)
    h = torch.randn(rows, width + 8, generator=g).to(BF).cuda()[:, :width]
    wr = (torch.randn(experts, width, generator=g) * 0.1).to(BF).cuda()
    br = torch.randn(experts, generator=g).cuda() if how == 0 else None
    ws = (torch.randn(width, generator=g) * 0.1).to(BF).cuda() if shared else None
    args = {} if how == 0 else dict(score_all=True, correction=torch.randn(experts, generator=g).cuda() * 0.01, weight_scale=1.5,
                                    renormalise=how == 2, groups=(4, 2) if how == 2 else None)
    top = 2

    def route(first, n):
        chosen = torch.full((n, top), -7, dtype=torch.int32, device="cuda")
        weight, gate = torch.full((n, top), float("nan"), device="cuda"), torch.full((n,), float("nan"), device="cuda") if shared else None
        ops.moe_route(chosen, weight, gate, h[first:first + n], wr, br, ws, n, top, **args)
        return chosen, weight, gate

    many = route(0, rows)
    for first in range(0, rows, 64):
        few = route(first, min(64, rows - first))
        for a, b in zip(many, few):
            assert a is None or torch.equal(a[first:first + 64], b)


@pytest.mark.parametrize("width", [3584, 1032, 100])
@pytest.mark.parametrize("identity", [0, 2])
def test_gather_and_combine(width, identity):
    """Widths that are and that are not whole 16-byte pieces."""
    from tessweave_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(width)
    rows, top, experts = 37, 3, 4
    h = torch.randn(rows, width + 8, generator=g).to(BF).cuda()[:, :width]
    chosen = torch.stack([torch.randperm(experts + identity, generator=g)[:top] for _ in range(rows)]).to(torch.int32).cuda()
    order, place, ends = sorted_pairs(ops, chosen, experts)
    xs = torch.full((rows * top, width), float("nan"), device="cuda", dtype=BF)
    ops.moe_gather(xs, h, order, rows * top, top)
    weight = torch.rand(rows, top, generator=g).cuda()
    shared, gate = torch.randn(rows, width, generator=g).to(BF).cuda(), torch.rand(rows, generator=g).cuda()
    out = torch.full((rows, width), float("nan"), device="cuda", dtype=BF)
    ops.moe_combine(out, xs, place, weight, shared, gate, rows, chosen=chosen, h=h, experts=experts, identity=identity)
    for p in range(rows * top):
        at = int(place[p])
        assert (at < 0) == (int(chosen.view(-1)[p]) >= experts)
        assert at < 0 or torch.equal(xs[at], h[p // top])
    want = weight.double().sum(1, keepdim=True) * h.double() + gate.double()[:, None] * shared.double()
    assert torch.allclose(out.double(), want, rtol=1.01 * 2 ** -8, atol=1e-5)           # one rounding to bf16, four fp32 terms of size 1
