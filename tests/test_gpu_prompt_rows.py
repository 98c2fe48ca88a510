"""Kernels of prompt steps that walk rows with wide accesses, against the kernels of few rows or plain torch."""
import pytest
import torch

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}


@pytest.mark.gpu
@pytest.mark.parametrize("out", ["float32", "bfloat16"])
@pytest.mark.parametrize("taps,unit_heads,unit_dim,channels", [(4, 3, 128, 640), (4, 2, 64, 576), (2, 3, 32, 160), (3, 0, 0, 516), (1, 5, 128, 640)])
@pytest.mark.parametrize("taps_first", [False, True])
def test_short_convolution_in_quads_of_channels(out, taps, unit_heads, unit_dim, channels, taps_first):
    """bf16 rows on 8-byte boundaries, many at once, give the bits of a block per row: requests of one row, shorter than the taps,
    ending inside and at the edge of eight rows, rows of no request, the last warp's channels behind the end, states moved on."""
    from tessweave_engine_b200.csrc import ops
    dev, keep, offset = torch.device("cuda"), taps - 1, 3
    g = torch.Generator().manual_seed(channels + taps)
    lengths = [1, 37, 2, 8, 1, 41, 3, 24]
    n, pad = sum(lengths), 5
    x = torch.randn(n + pad, channels + 4, generator=g).bfloat16().to(dev)
    w = torch.randn(taps, channels, generator=g).mul(0.5).to(dev).t()
    if taps_first:
        w = w.contiguous()
    bias = torch.randn(channels, generator=g).to(dev)
    state = torch.randn(len(lengths) + 1, offset + channels * keep, generator=g).to(dev)
    slots = torch.randperm(len(lengths), generator=g).to(torch.int32).to(dev)
    kw = dict(unit_heads=unit_heads, unit_dim=unit_dim, scaled_heads=min(1, unit_heads), head_scale=0.25, unit_eps=1e-6, bias=bias)

    def step(rows, lens, slots, st):
        res = torch.full((rows.shape[0], channels), 7.0, device=dev, dtype=DTYPES[out])
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)      # noqa: E731
        seq = i32([i for i, m in enumerate(lens) for _ in range(m)] + [-1] * (rows.shape[0] - sum(lens)))
        ops.short_conv(res, rows, w, st, offset, seq, slots, i32([sum(lens[:i]) for i in range(len(lens))]), rows.shape[0],
                       move_single=i32(lens), **kw)
        return res

    moved, want_state = state.clone(), state.clone()
    got = step(x, lengths, slots, moved)
    want, at = [], 0
    for i, m in enumerate(lengths):
        want.append(step(x[at:at + m], [m], slots[i:i + 1].contiguous(), want_state))
        at += m
    assert torch.equal(got[:n], torch.cat(want)) and torch.equal(moved, want_state)
    assert bool((got[n:] == 7.0).all()), "rows of no request were written"


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows,heads,dim,act,with_den,odd", [(1, 1, 32, 1, False, 0), (7, 3, 64, 2, True, 0), (65, 14, 128, 1, True, 0),
                                                            (33, 5, 128, 0, False, 0), (9, 3, 48, 1, True, 0), (9, 3, 64, 2, True, 1)])
def test_head_norm_and_gate(dtype, rows, heads, dim, act, with_den, odd):
    """Heads served with wide accesses (32, 64, 128 values on 16-byte boundaries) and the others: a value of the result is the product
    of five numbers, each rounded a few times in 32 bits, and rounded once to its type."""
    from tessweave_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(rows * 7 + dim)
    width = heads * dim
    raw = torch.randn(rows, width, generator=g) * 3
    den = torch.rand(rows, heads, generator=g) + 0.5 if with_den else None
    weight = torch.randn(width, generator=g)
    gate = torch.randn(rows, width + 4 + odd, generator=g).to(DTYPES[dtype])[:, odd:odd + width] if act else None
    dev = lambda t: None if t is None else t.cuda()     # noqa: E731
    out = torch.zeros(rows, width + 4 + odd, dtype=DTYPES[dtype], device="cuda")[:, :width]
    gate_dev = None
    if gate is not None:
        whole = torch.zeros(rows, width + 4 + odd, dtype=DTYPES[dtype], device="cuda")
        gate_dev = whole[:, odd:odd + width]
        gate_dev.copy_(gate)
    ops.head_norm_gate(out, dev(raw), dev(den), dev(weight), gate_dev, act, 1e-6, rows, heads, dim)
    o = raw.double().view(rows, heads, dim)
    if den is not None:
        o = o / den.double()[:, :, None]
    y = (o / torch.sqrt(o.square().mean(-1, keepdim=True) + 1e-6)).view(rows, width) * weight.double()
    if act:
        gd = gate.double()
        y = y * (torch.sigmoid(gd) * (gd if act == 1 else 1.0))
    got = out.cpu().double()
    bound = 2.0 ** -8 if dtype == "bfloat16" else 64 * 2.0 ** -24      # (half a step of the result's type, with room for the chain)
    assert bool(((got - y).abs() <= bound * y.abs() + 1e-30).all())
