"""32-bit products on the tensor cores against 64 bits: every shape of the kernel at the edges of its tiles, slices of K that
are short or empty, results that depend on no other row, and operands that are not finite."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from tiny_llm_b200 import ops
    return ops


def bound(a, w):
    """What the sums may be away from 64 bits, in sizes |a w| added up: the product left out (2^-34); the large accumulator, four
    additions of 16 products per block of 64 with at most two units of truncation of the block's sizes each; the small ones,
    2^-8 of the sizes (or less), with eight additions per 16 values of k; an addition to the running sum per block, two for the
    small ones and three for the slices."""
    k = a.shape[1]
    size = a.double().abs() @ w.double().abs().T
    return (2.0 ** -34 + 4 * 2.0 ** -22 + 8 * math.ceil(k / 16) * 2.0 ** -30 + (math.ceil(k / 64) + 5) * 2.0 ** -24) * size


@pytest.mark.parametrize("n,k", [(512, 2048), (4128, 2048), (32, 32768), (544, 2080), (2048, 3040), (32000, 2048), (1056, 2208)])
def test_rows_of_every_count_are_near_64_bits_and_depend_on_no_other_row(ops, n, k):
    """(2,080: 33 blocks, the last a half, in eight slices of five, the last empty; 3,040: half a block at the end.)"""
    g = torch.Generator(device=DEV).manual_seed(n + k)
    rows = torch.randn(1300, k + 4, generator=g, device=DEV)[:, :k]
    w = torch.randn(n, k, generator=g, device=DEV) * torch.rand(n, 1, generator=g, device=DEV)
    assert ops._f32_tc_ok(rows, w)
    want, most = rows.double() @ w.double().T, bound(rows, w)
    whole = None
    for m in (1300, 1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 256, 700):
        out, acc = torch.full((m, n + 4), 7.0, device=DEV), torch.full((m, n), 0.5, device=DEV)
        ops.linear(rows[:m], w, out[:, :n])
        ops.linear(rows[:m], w, acc, accumulate=True)
        whole = out[:, :n].clone() if whole is None else whole
        assert torch.equal(out[:, :n], whole[:m]) and bool((out[:, n:] == 7.0).all()), m
        assert torch.equal(acc, whole[:m] + 0.5), m
    ops.check_status()
    assert bool(((whole - want).abs() <= most).all())


def test_the_order_of_the_sums_follows_from_the_weight_alone(ops, monkeypatch):
    """Neither the switch of the bfloat16 path's slices nor the number of SMs moves a bit."""
    g = torch.Generator(device=DEV).manual_seed(5)
    for n, k in ((2048, 2048), (8192, 2048)):
        a, w = torch.randn(24, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV)
        outs = []
        for split, sms in ((True, 148), (False, 148), (True, 40), (True, 160)):
            monkeypatch.setattr(ops, "split_k", split)
            monkeypatch.setattr(ops, "sm_count", lambda *_, sms=sms: sms)
            out = torch.empty(24, n, device=DEV)
            ops.linear(a, w, out)
            outs.append(out)
        assert all(torch.equal(o, outs[0]) for o in outs)


def test_a_single_product_is_as_near_as_one_rounding(ops):
    """Rows of one value each: eight partial products leave 2^-34 out, and the sum is rounded once (2^-24).  With parts that are cut
    instead of rounded the first pair is 4.7e-7 off."""
    g = torch.Generator(device=DEV).manual_seed(1)
    n, k = 512, 2048
    for m in (16, 200):
        a, w = torch.zeros(m, k, device=DEV), torch.zeros(n, k, device=DEV)
        a[:, 77] = torch.randn(m, generator=g, device=DEV)
        w[:, 77] = torch.randn(n, generator=g, device=DEV)
        a[0, 77] = w[0, 77] = 1 + 2.0 ** -7 - 2.0 ** -23
        out = torch.empty(m, n, device=DEV)
        ops.linear(a, w, out)
        want = a[:, 77:78].double() @ w[:, 77:78].double().T
        assert bool(((out - want).abs() <= want.abs() * (2.0 ** -24 + 2.0 ** -34)).all())
    ops.check_status()


@pytest.mark.parametrize("n", [512, 32000])
@pytest.mark.parametrize("values", [1, 2, 4, 8, 16])
def test_rows_of_few_values_are_as_near_as_one_chain_of_fmaf(ops, n, values, monkeypatch):
    """A chain rounds once per value.  The tensor cores' sums are rounded once per block with values and once more per slice with
    values (n = 512: eight slices), so two to four values in slices of their own come out up to a sixth further off."""
    g = torch.Generator(device=DEV).manual_seed(values + n)
    m, k, away = 400, 2048, {}
    a = torch.zeros(m, k, device=DEV)
    where = torch.rand(m, k, generator=g, device=DEV).argsort(1)[:, :values]
    a.scatter_(1, where, torch.randn(m, values, generator=g, device=DEV))
    w = torch.randn(n, k, generator=g, device=DEV)
    want, size = a.double() @ w.double().T, (a.double().abs() @ w.double().abs().T).clamp_min(1e-30)
    for tc in (True, False):
        monkeypatch.setattr(ops, "linear_f32_tc", tc)
        out = torch.empty(m, n, device=DEV)
        ops.linear(a, w, out)
        away[tc] = float(((out - want) / size).square().mean().sqrt())
    assert away[True] <= away[False] * 1.2, away


@pytest.mark.parametrize("n,k", [(2048, 2048), (2048, 5632), (11264, 2048)])
def test_no_further_from_64_bits_than_one_chain_of_fmaf(ops, n, k, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(k)
    a, w = torch.randn(200, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV) * 0.02
    for x in (a, a.abs() + 0.5):                  # sums that wander, and sums that grow (with weights of one sign)
        y = w if x is a else w.abs()
        want, away = x.double() @ y.double().T, {}
        for tc in (True, False):
            monkeypatch.setattr(ops, "linear_f32_tc", tc)
            out = torch.empty(200, n, device=DEV)
            ops.linear(x, y, out)
            away[tc] = float((out - want).norm() / want.norm())
        assert away[True] <= away[False], away


@pytest.mark.parametrize("m", [8, 40, 130])
def test_operands_of_every_size_are_split_exactly(ops, m):
    """Rows of 1e-25 to the smallest subnormal numbers against weights of 1e-6 to 1e20, and rows near the largest numbers against
    small weights: the bound is the same, beside the last place of a subnormal result.  (The largest are made as chains of
    fmaf, 2^-24 per value.)"""
    g = torch.Generator(device=DEV).manual_seed(m)
    n, k = 1024, 2048
    a, w = torch.randn(m, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV)
    sizes = torch.tensor([1e-25, 1e-30, 1e-33, 1e-35, 1e-36, 2e-38, 1e-40, 1e20, 1e30, 1e32, 1e36], dtype=torch.float64, device=DEV)
    a = (a.double() * sizes[torch.arange(m, device=DEV) % len(sizes)][:, None]).float()
    w = w * torch.tensor([1.0, 1e-6, 1e20, 1e-3], device=DEV)[torch.arange(n, device=DEV) % 4][:, None]
    out = torch.empty(m, n, device=DEV)
    ops.linear(a, w, out)
    want = a.double() @ w.double().T
    size = a.double().abs() @ w.double().abs().T
    here = size < 1e38                     # (no partial sum of a chain overflows)
    most = torch.where(a.abs().amax(1, keepdim=True) > 1e19, size * k * 2.0 ** -24, bound(a, w)) + 2.0 ** -149
    assert bool(((out - want).abs() <= most)[here].all()) and int(here.sum()) > m * n // 2
    ops.check_status()


def test_operands_that_are_not_finite_give_what_one_chain_of_fmaf_gives(ops, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(3)
    n, k = 1024, 2048
    a, w = torch.randn(130, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV)
    a[3, 7], a[40, 900], a[77, 1], a[100, 5] = math.inf, -math.inf, math.nan, 3.4e38
    w[9, 40], w[600, 3], w[700, 5] = math.inf, math.nan, 3.0
    a[120], w[33] = 1e-30, 1e-30           # sums below the normal range
    outs = {}
    for tc in (True, False):
        monkeypatch.setattr(ops, "linear_f32_tc", tc)
        for m in (130, 8):
            out = torch.empty(m, n, device=DEV)
            ops.linear(a[:m], w, out)
            outs[tc, m] = out
    for m in (130, 8):
        got, want = outs[True, m], outs[False, m]
        odd = ~torch.isfinite(want)
        assert bool(odd.any()) and torch.equal(torch.isfinite(got), ~odd)
        assert torch.equal(got[odd].nan_to_num(nan=1.5), want[odd].nan_to_num(nan=1.5))
        size = a[:m].nan_to_num(0, 0, 0).abs().double() @ w.nan_to_num(0, 0, 0).abs().double().T
        assert bool(((got.double() - want.double()).abs()[~odd] <= (size * k * 2.0 ** -23 + 1e-37)[~odd]).all())


@pytest.mark.parametrize("m", [8, 300])
def test_rows_of_nan_take_no_longer_than_others(ops, m):
    """(A chain of 2,048 fmaf per element, one thread each, took many times the product.)"""
    g = torch.Generator(device=DEV).manual_seed(m)
    a, w, took = torch.randn(m, 2048, generator=g, device=DEV), torch.randn(11264, 2048, generator=g, device=DEV), {}
    out = torch.empty(m, 11264, device=DEV)
    for kind, rows in (("finite", a), ("nan", torch.full_like(a, math.nan))):
        times = []
        for _ in range(6):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            for _ in range(4):
                ops.linear(rows, w, out)
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end))
        took[kind] = min(times)
    assert bool(out.isnan().all()) and took["nan"] < 1.5 * took["finite"], took
