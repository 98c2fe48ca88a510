"""The recurrences of prompt portions in chunks, against the same recurrence token by token in 64 bits, at the edges of the
chunks of 64 tokens, behind a state, beside short portions."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LENS = [193, 1, 32, 256, 31, 127]               # below 32 rows a request is left to the token kernel
SLOTS = [3, 0, 6, 1, 5, 2]


def operands(rule, heads, dk, dv, rot, lens, seed=0, decay=None):
    g = torch.Generator().manual_seed(seed)
    n = sum(lens)
    bf = torch.bfloat16
    wide = torch.randn(n, heads * (2 * dk + dv) + 8, generator=g).to(bf).cuda()
    o = {"q": wide[:, :heads * dk], "k": wide[:, heads * dk:2 * heads * dk], "v": wide[:, 2 * heads * dk:2 * heads * dk + heads * dv]}
    held = [7 * i for i in range(len(lens))]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")          # noqa: E731
    o["positions"] = i32([h + t for m, h in zip(lens, held) for t in range(m)])
    o["start"], o["len"], o["slot"] = i32([sum(lens[:i]) for i in range(len(lens))]), i32(lens), i32(SLOTS[:len(lens)])
    if rule == "delta":                         # prepared rows: fp32, q and k of unit length, two value heads to a q/k head
        unit = lambda m: torch.nn.functional.normalize(torch.randn(n, m, dk, generator=g), dim=-1).view(n, -1)       # noqa: E731
        half = heads // 2
        rows = torch.cat((unit(half) * dk ** -0.5, unit(half), torch.randn(n, heads * dv, generator=g)), 1).cuda()
        o["q"], o["k"], o["v"] = rows[:, :half * dk], rows[:, half * dk:heads * dk], rows[:, heads * dk:]
    cols = dv + (1 if rule == "mlstm" else 0)
    state = torch.randn(7, heads * (dk * cols + (1 if rule == "mlstm" else 0)) + 5, generator=g)
    if rule == "mlstm":
        state[:, :-5].view(7, heads, -1)[:, :, -1] = torch.randn(7, heads, generator=g) * 3
        # gates from gentle to violent: memories of hundreds of tokens, and ones that are wiped out by a single token
        pre = torch.randn(n, 2 * heads, generator=g) * torch.linspace(1, 12, heads).repeat(2)
        o["args"] = {"pre": pre.cuda(), "p0": torch.cat([torch.zeros(heads), torch.full((heads,), 2.0)]).cuda(), "q_scale": dk ** -0.5,
                     "cap": 15.0}
    elif rule == "delta":
        # decays from none worth mentioning to memories that are gone within a token, write strengths on both sides of a half
        pre = torch.randn(n, 2 * heads, generator=g) * torch.linspace(1, 6, heads).repeat(2)
        o["args"] = {"pre": pre[:, heads:].contiguous().cuda(), "write_pre": pre.cuda(), "p0": torch.linspace(-5, 1, heads).cuda(),
                     "p1": torch.randn(heads, generator=g).cuda(), "qk_group": 2}
    else:
        decay = decay if decay is not None else [1.0 - 2.0 ** -(h + 1) for h in range(heads)]
        o["args"] = {"p0": torch.tensor(decay, dtype=torch.float32).cuda(), "k_scale": dk ** -0.5}
        if rot:
            o["args"].update(inv_freq=(100.0 ** (-torch.arange(0, rot, 2) / rot)).float().cuda(), rot_dims=rot)
    o["state"] = state.cuda()
    return o


def token_by_token(rule, o, heads, dk, dv, rot, a, m, slot):
    """(outputs, denominators, state) of rows a .. a + m - 1 in 64 bits."""
    q, k = (o[x][a:a + m].double().cpu().view(m, -1, dk) for x in "qk")
    v = o["v"][a:a + m].double().cpu().view(m, heads, dv)
    st = o["state"][slot, :-5].double().cpu().view(heads, -1)
    out, den = torch.zeros(m, heads, dv, dtype=torch.float64), torch.zeros(m, heads, dtype=torch.float64)
    if rule == "delta":
        S, A = st.view(heads, dk, dv).clone(), {x: t.double().cpu() for x, t in o["args"].items() if x != "qk_group"}
        q, k = q.repeat_interleave(2, 1), k.repeat_interleave(2, 1)
        keep = torch.exp(-torch.exp(A["p0"]) * torch.nn.functional.softplus(A["pre"][a:a + m, :heads] + A["p1"], threshold=700.0))
        beta = torch.sigmoid(A["write_pre"][a:a + m, :heads])
        for t in range(m):
            S = keep[t][:, None, None] * S
            u = beta[t][:, None] * (v[t] - torch.einsum("hij,hi->hj", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None]
            out[t] = torch.einsum("hij,hi->hj", S, q[t])
        return out, den, S.reshape(-1)
    if rule == "retention":
        S = st.view(heads, dk, dv).clone()
        if rot:
            # the angle is an fp32 product in the kernels; what follows from it is taken from there
            ang = (o["positions"][a:a + m].cpu().float()[:, None] * o["args"]["inv_freq"].cpu()).double()
            c, s = ang.cos()[:, None], ang.sin()[:, None]
            turn = lambda x: torch.cat((x[..., :rot // 2] * c - x[..., rot // 2:rot] * s,      # noqa: E731
                                        x[..., rot // 2:rot] * c + x[..., :rot // 2] * s, x[..., rot:]), -1)
            q, k = turn(q), turn(k)
        k = k * dk ** -0.5
        d = o["args"]["p0"].double().cpu()[:, None, None]
        for t in range(m):
            S = d * S + k[t][:, :, None] * v[t][:, None]
            out[t] = torch.einsum("hij,hi->hj", S, q[t])
        return out, den, S.reshape(-1)
    S, top = st[:, :-1].view(heads, dk, dv + 1).clone(), st[:, -1].clone()
    q = q * dk ** -0.5
    v = torch.cat((v, torch.ones(m, heads, 1, dtype=torch.float64)), 2)
    pre, bias = o["args"]["pre"][a:a + m].double().cpu(), o["args"]["p0"].double().cpu()
    gi = 15 * torch.tanh((pre[:, :heads] + bias[:heads]) / 15)
    gf = torch.nn.functional.logsigmoid(15 * torch.tanh((pre[:, heads:] + bias[heads:]) / 15))
    for t in range(m):
        new = torch.maximum(gf[t] + top, gi[t])
        S = torch.exp(gf[t] + top - new)[:, None, None] * S + (torch.exp(gi[t] - new)[:, None] * k[t])[:, :, None] * v[t][:, None]
        top = new
        o_t = torch.einsum("hij,hi->hj", S, q[t])
        out[t], den[t] = o_t[:, :dv], torch.maximum(o_t[:, dv].abs(), torch.exp(-top)) + 1e-6
    return out, den, torch.cat((S.reshape(heads, -1), top[:, None]), 1).reshape(-1)


def run(rule, o, heads, dk, dv, chunks, write=True, lens=LENS):
    from tessweave_engine_b200.csrc import ops
    mode = {"mlstm": ops.RECURRENCE_MLSTM, "retention": ops.RECURRENCE_RETENTION, "delta": ops.RECURRENCE_DELTA}[rule]
    n = o["q"].shape[0]
    out, den = torch.full((n, heads * dv), -7.0, device="cuda"), torch.full((n, heads), -7.0, device="cuda")
    state = o["state"].clone()
    common = (out, den if rule == "mlstm" else None, o["q"], o["k"], o["v"], state, o["positions"], o["slot"], o["start"], o["len"], len(lens),
              heads, dk, dv)
    if chunks and rule == "delta":
        count = ops.recurrence_chunk_count(n, len(lens)) * ops.delta_chunk_floats(heads, 2, dk, dv)
        ops.delta_chunks(out, o["q"], o["k"], o["v"], state, *common[7:], max(lens), torch.full((count,), float("nan"), device="cuda"), write,
                         **o["args"])
    elif chunks:
        count = ops.recurrence_chunk_count(n, len(lens))
        nan = lambda k, dt=torch.float32: torch.full((k,), float("nan"), device="cuda", dtype=dt)         # noqa: E731
        ops.recurrence_chunks(mode, *common, max(lens), nan(count * heads * dk * (dv + 1)), nan(count * heads * 2, torch.float64),
                              nan(count * heads), write, **o["args"])
    else:
        ops.linear_recurrence(mode, *common, write, max_q_len=max(lens), **o["args"])
    return out.view(n, heads, dv).cpu().double(), den.cpu().double(), state.cpu()


def distance(got, want):
    return float((got - want).norm() / want.norm().clamp_min(1e-30))


@pytest.mark.parametrize("rule,heads,dk,dv,rot", [("mlstm", 3, 128, 128, 0), ("mlstm", 2, 64, 128, 0), ("mlstm", 5, 64, 64, 0),
                                                  ("mlstm", 2, 32, 64, 0), ("retention", 3, 128, 128, 128), ("retention", 2, 64, 64, 0),
                                                  ("retention", 4, 128, 64, 64), ("retention", 2, 32, 128, 32),
                                                  ("delta", 4, 128, 128, 0), ("delta", 6, 64, 64, 0), ("delta", 2, 64, 128, 0),
                                                  ("delta", 2, 128, 64, 0)])
def test_chunks_against_tokens(rule, heads, dk, dv, rot):
    """The chunks' error against 64 bits is that of the token kernel or below it.  A quarter more is allowed for chance, and the
    least that 32 bits leave: 1e-7 in sums; with mLSTM's gates, numbers of up to 15 evaluated in 32 bits (an error of up to
    15 x 2^-23 in an exponent, where one token may be all that counts), a third of that, 6e-7.  Short requests, other slots and
    what lies behind the heads are left alone."""
    least = 6e-7 if rule == "mlstm" else 1e-7
    o = operands(rule, heads, dk, dv, rot, LENS)
    got, token = run(rule, o, heads, dk, dv, True), run(rule, o, heads, dk, dv, False)
    a = 0
    for m, slot in zip(LENS, SLOTS):
        if m < 32:
            assert torch.all(got[0][a:a + m] == -7.0) and torch.equal(got[2][slot], o["state"][slot].cpu())
        else:
            want = token_by_token(rule, o, heads, dk, dv, rot, a, m, slot)
            pairs = [(r[0][a:a + m], r[2][slot, :-5].double()) for r in (got, token)]
            names = [("outputs", 0, want[0]), ("state", 1, want[2])]
            if rule == "mlstm":
                # the memory is kept divided by e^m, whatever 32-bit m the kernel has: compared as it stands for the exact m
                w = want[2].view(heads, -1)
                exact = lambda st: (st.view(heads, -1) * torch.exp(st.view(heads, -1)[:, -1:] - w[:, -1:]))[:, :-1]     # noqa: E731
                assert float((pairs[0][1].view(heads, -1)[:, -1] - w[:, -1]).abs().max()) < 4e-6             # |m| up to 15, some 2^-24 of it
                pairs, names[1] = [(p[0], exact(p[1])) for p in pairs], ("state", 1, w[:, :-1])
                pairs = [(*p, r[1][a:a + m]) for p, r in zip(pairs, (got, token))]
                names.append(("denominators", 2, want[1]))
            for name, i, w in names:
                mine, theirs = distance(pairs[0][i], w), distance(pairs[1][i], w)
                assert mine <= max(1.25 * theirs, least), f"{name} of {m} rows: {mine:.2e}, token by token {theirs:.2e}"
        assert torch.equal(got[2][slot, -5:], o["state"][slot, -5:].cpu())
        a += m
    assert torch.equal(got[2][4], o["state"][4].cpu())                         # nobody's slot
    again = run(rule, o, heads, dk, dv, True, write=False)
    assert torch.equal(again[0], got[0]) and torch.equal(again[2], o["state"].cpu())


@pytest.mark.parametrize("decay", [[0.0, 1.0], [1.25, -0.5]])
def test_decays_at_the_edges(decay):
    """No memory, a memory that never fades, one that grows, one that changes its sign."""
    o = operands("retention", 2, 64, 64, 0, [130, 1, 128], decay=decay)
    got = run("retention", o, 2, 64, 64, True, lens=[130, 1, 128])
    for a, m, slot in ((0, 130, 3), (131, 128, 6)):
        want = token_by_token("retention", o, 2, 64, 64, 0, a, m, slot)
        for h in range(2):
            # 32-bit sums of 64 terms and a carried sum: some 2^-24 x 8 of what was added up
            assert distance(got[0][a:a + m, h], want[0][:, h]) < 5e-7
            assert distance(got[2][slot, :-5].double().view(2, -1)[h], want[2].view(2, -1)[h]) < 5e-7


@pytest.mark.parametrize("rule", ["mlstm", "retention", "delta"])
def test_a_token_does_not_reach_those_before_it(rule):
    """A value that is infinite or not a number spoils its own token's column and later ones, nothing earlier."""
    lens = [321, 1, 128, 256]
    o = operands(rule, 2, 64, 64, 0, lens)
    clean = run(rule, o, 2, 64, 64, True, lens=lens)
    o["v"][70, 5], o["v"][72, 64 + 9] = float("inf"), float("nan")              # heads 0 and 1 of the first request
    got = run(rule, o, 2, 64, 64, True, lens=lens)
    same = torch.ones(clean[0].shape, dtype=torch.bool)
    same[70:321, 0, 5] = same[72:321, 1, 9] = False
    assert torch.equal(got[0][same], clean[0][same])
    assert not torch.isfinite(got[0][70:321, 0, 5]).any() and torch.isnan(got[0][72:321, 1, 9]).all()
