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
    """What the sums may be away from 64 bits: the three partial products left out (2^-24 each of |a w| at most), three
    accumulators that add 16 products at a time (4 + 8 + 12 additions per block of 64, of which the last twenty are 2^-7
    smaller) with at most two units of truncation of the block's |a w| each, and three additions per block to the running
    sum."""
    k = a.shape[1]
    size = a.double().abs() @ w.double().abs().T
    return (3 * 2.0 ** -24 + (4 + 20 * 2.0 ** -7) * 2.0 ** -22 + (3 * math.ceil(k / 64) + 8) * 2.0 ** -24) * size


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
