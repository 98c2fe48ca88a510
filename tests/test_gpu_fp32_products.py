"""32-bit products on the tensor cores (three bf16 terms per number) against 64 bits."""
import pytest
import torch


def ops():
    from tessweave_engine_b200.csrc import ops as o
    from tessweave_engine_b200.parts.linear import configure_matmul_precision
    configure_matmul_precision()
    return o


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,x_more,out_more", [(1, 1, 4, 0, 0), (128, 128, 64, 0, 0), (129, 127, 68, 4, 1), (300, 260, 128, 0, 4),
                                                  (257, 384, 132, 8, 0), (640, 1152, 896, 0, 0), (200, 130, 1000, 4, 2)])
@pytest.mark.parametrize("spread", [0, 30])
def test_product(m, n, k, x_more, out_more, spread):
    """Edges of tiles, of 64 values of k and of the wide stores; ``spread``: numbers over 60 powers of two.  An MMA aligns its 16
    products and the sum so far to the largest of them and cuts each off at 2^-24 of that (17 x 2^-24 of the sum of sizes); four of
    them follow one another, the smaller products' sums and what is left out lie below: 2^-17 of the sum of the products' sizes
    bounds it all.  With numbers of one size the error as a whole is no larger than that of plain 32-bit sums."""
    o = ops()
    g = torch.Generator().manual_seed(m + k)
    make = lambda r, c: torch.randn(r, c, generator=g) * torch.exp2(torch.randint(-spread, spread + 1, (r, c), generator=g).float())   # noqa: E731
    x, w = make(m, k), make(n, k)
    xd = torch.zeros(m, k + x_more, device="cuda")[:, :k]
    xd.copy_(x)
    out = torch.full((m, n + out_more), 7.0, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    o.gemm_fp32(out[:, :n], xd, w.cuda(), m, status)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert bool(((out[:, :n].cpu().double() - want).abs() <= 2.0 ** -17 * size).all())
    if k >= 128 and not spread:
        plain = torch.mm(x.cuda(), w.cuda().T).cpu().double()
        assert float((out[:, :n].cpu().double() - want).norm()) <= float((plain - want).norm())
    assert bool((out[:, n:] == 7.0).all()) and int(status) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("k", [512, 896, 1536])
@pytest.mark.parametrize("spread", [4, 15, 30])
def test_numbers_of_many_sizes(k, spread):
    """At a size that goes through here, with numbers spread over 8 to 60 powers of two: the error as a whole is no larger than that of plain
    32-bit sums (0.2 to 0.85 of it)."""
    o, m, n = ops(), 640, 1152
    g = torch.Generator().manual_seed(k + spread)
    make = lambda r: torch.randn(r, k, generator=g) * torch.exp2(torch.randint(-spread, spread + 1, (r, k), generator=g).float())   # noqa: E731
    x, w, out = make(m).cuda(), make(n).cuda(), torch.empty(m, n, device="cuda")
    assert o.prefer_gemm_fp32(m, n, k)
    o.gemm_fp32(out, x, w, m, torch.zeros(1, dtype=torch.int32, device="cuda"))
    want = x.double() @ w.double().T
    assert float((out.double() - want).norm()) <= float((torch.mm(x, w.T).double() - want).norm())


@pytest.mark.gpu
@pytest.mark.parametrize("small", ["x", "w"])
@pytest.mark.parametrize("power", [-100, -112, -120, -126, -135])
def test_the_smallest_numbers(small, power):
    """Operands whose last bits lie below what a bf16 number holds, down to numbers that have lost bits themselves: the error is no larger
    than that of plain 32-bit sums."""
    o, m, n, k = ops(), 130, 260, 512
    g = torch.Generator().manual_seed(-power)
    make = lambda rows, tiny: (torch.randn(rows, k, generator=g).double() * 2.0 ** (power if tiny else 3)).float()      # noqa: E731
    x, w = make(m, small == "x"), make(n, small == "w")
    out, status = torch.empty(m, n, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    o.gemm_fp32(out, x.cuda(), w.cuda(), m, status)
    want, plain = x.double() @ w.double().T, torch.mm(x.cuda(), w.cuda().T).cpu().double()
    assert float((out.cpu().double() - want).norm()) <= float((plain - want).norm()) and int(status) == 0


@pytest.mark.gpu
def test_numbers_without_three_terms():
    """Infinities, NaN and numbers above the largest bf16 give what plain 32-bit sums give, and reach no other row or column."""
    o = ops()
    g = torch.Generator().manual_seed(3)
    x, w = torch.randn(150, 128, generator=g), torch.randn(140, 128, generator=g)
    x[3, 5], x[7, 9], x[20, 1], x[21] = float("inf"), float("nan"), 3.4e38, 0.0
    w[11, 3], w[:, 1] = -float("inf"), 0.5
    x[21, 1] = 3.4e38
    out = torch.empty(150, 140, device="cuda")
    o.gemm_fp32(out, x.cuda(), w.cuda(), 150, torch.zeros(1, dtype=torch.int32, device="cuda"))
    want = x.double() @ w.double().T
    got = out.cpu().double()
    finite = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    assert bool((torch.sign(got) == torch.sign(want))[torch.isinf(want)].all())
    size = x.double().nan_to_num(0, 0, 0).abs() @ w.double().nan_to_num(0, 0, 0).abs().T
    assert bool(((got - want).abs() <= 2.0 ** -17 * size)[finite].all())


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,x_more", [(333, 260, 132, 4), (128, 128, 32, 0), (130, 390, 1000, 0), (5, 3, 4, 0)])
def test_many_sums_that_are_not_finite(m, n, k, x_more):
    """Rows of x and of w with infinities and NaN throughout, at both ends and at edges of tiles: every sum that is not finite in 64 bits
    is the same kind of number here, every other one within the bound, and nothing behind the last row or column is written."""
    o = ops()
    g = torch.Generator().manual_seed(m)
    x, w = torch.randn(m, k, generator=g), torch.randn(n, k, generator=g)
    bad = (float("inf"), -float("inf"), float("nan"))
    for t, step in ((x, 3), (w, 41)):
        for i in {*range(0, t.shape[0], step), t.shape[0] - 1}:
            t[i, (i * 7) % k] = bad[i % 3]
    w[0, :: 2] = 0.0                            # (an infinity times zero is no number)
    xd = torch.zeros(m, k + x_more, device="cuda")[:, :k]
    xd.copy_(x)
    out, status = torch.full((m + 1, n), 7.0, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    o.gemm_fp32(out[:m], xd, w.cuda(), m, status)
    want, got = x.double() @ w.double().T, out[:m].cpu().double()
    finite = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    clean = lambda t: t.double().nan_to_num(0, 0, 0).abs()      # noqa: E731
    assert bool(((got - want).abs() <= 2.0 ** -17 * (clean(x) @ clean(w).T))[finite].all())
    assert bool((out[m] == 7.0).all()) and int(status) == 0


@pytest.mark.gpu
def test_numbers_that_are_not_finite_cost_little():
    """A matrix full of NaN (a model that has diverged): a few times the product's time, here at most 20 times; sum by sum, by one thread
    for a row, it was hundreds of times."""
    o = ops()
    m, n, k = 777, 896, 4864
    x, w, out = torch.randn(m, k, device="cuda"), torch.randn(n, k, device="cuda"), torch.empty(m, n, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def us(rows):
        times = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            o.gemm_fp32(out, rows, w, m, status)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b) * 1e3)
        return min(times)

    plain = us(x)
    worst = us(torch.full_like(x, float("nan")))
    assert bool(torch.isnan(out).all()) and worst < 20 * plain, (plain, worst)
    print(f"finite {plain:.1f} us, NaN {worst:.1f} us")


@pytest.mark.gpu
def test_which_products_and_what_is_refused():
    o = ops()
    assert o.prefer_gemm_fp32(777, 896, 896) and not o.prefer_gemm_fp32(512, 1152, 896) and not o.prefer_gemm_fp32(64, 151936, 896)
    x, w = torch.zeros(130, 66, device="cuda"), torch.zeros(128, 66, device="cuda")
    assert not o.gemm_fp32_supported(x, w) and not o.gemm_fp32_supported(x.bfloat16(), w.bfloat16())
    with pytest.raises(Exception, match="gemm_fp32"):
        o.gemm_fp32(torch.zeros(130, 128, device="cuda"), x, w, 130, torch.zeros(1, dtype=torch.int32, device="cuda"))
