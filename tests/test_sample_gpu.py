"""Sampler kernel where its slices, clusters, counters, segments and key ranges have edges, against a host restatement of its
fixed-point arithmetic."""
import numpy as np
import pytest
import torch

from ferrl_b200.sampler import uniforms_for_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,V,dtype,std,top_p,T,pad", [
    (1, 1, torch.bfloat16, 1.0, 0.9, 1.0, 0), (3, 7, torch.float32, 1.0, 0.5, 0.7, 0),         # less than a group
    (2, 8191, torch.bfloat16, 2.0, 0.95, 1.0, 1), (2, 8192, torch.float32, 3.0, 0.8, 1.2, 4),   # one CTA; ragged and strided rows
    (1, 65537, torch.bfloat16, 2.5, 0.95, 1.0, 0), (5, 50257, torch.float32, 2.5, 0.9, 1.0, 3),  # clusters with a short last slice
    (130, 151936, torch.bfloat16, 2.5, 0.95, 1.0, 0), (4, 262144, torch.float32, 2.5, None, 0.7, 0),
    (4, 32000, torch.bfloat16, 0.0, 0.3, 1.0, 0), (4, 32000, torch.bfloat16, 40.0, 0.999, 1.0, 0),   # all equal; almost all mass on one
    (2, 9000, torch.bfloat16, 0.01, 0.5, 1.0, 0), (2, 9000, torch.float32, 1e-3, 0.5, 1.0, 0),       # the cut around zero: widest key range
    (2, 20000, torch.bfloat16, 300.0, 0.9, 100.0, 0), (2, 20000, torch.bfloat16, 1e-4, 0.9, 1.0, 0),  # values without a counter: large, small
    (1, 1400000, torch.bfloat16, 2.0, 0.9, 1.0, 0),                                                  # slices of many elements
])
def test_draws_match_the_fixed_point_oracle(rows, V, dtype, std, top_p, T, pad):
    from ferrl_b200.ops import cuda as Cc
    g = torch.Generator(device="cuda").manual_seed(rows * V)
    x = (torch.randn(rows, V + pad, generator=g, device="cuda") * std + (std == 0)).to(dtype)[:, :V]
    if V > 100:
        x[:, 5:50] = float("-inf")                                           # masked vocabulary entries
    ids = torch.randint(0, 1 << 40, (rows,), generator=g, device="cuda")
    u = uniforms_for_rows(11, ids.cpu(), 3).double().numpy()
    tok, lp = (t.cpu().numpy() for t in Cc.sample_top_p(x, 11, ids, 3, T, top_p, None))
    xs = x.double().cpu().numpy()
    for r in range(rows):
        # the device's exponential and its 2^-40 truncation move every mass by 1e-5 of it (arguments down to -90), which
        # moves the cut and the drawn point by as much of the whole; lp additionally rounds a float32 logarithm
        e = np.exp((xs[r] - xs[r].max()) / T)
        keep = np.ones(V, bool)
        eps = 2e-5
        if top_p is not None:
            order = np.argsort(-e, kind="stable")
            cum = e[order].cumsum()
            at = lambda p: e[order[min(V - 1, int(np.searchsorted(cum, p * cum[-1])))]]  # noqa: E731
            lo, hi = at(min(1.0, top_p + eps)), at(top_p - eps)
            assert e[tok[r]] >= lo * (1 - eps)
            keep = e >= lo * (1 - eps)
            surely = (e >= hi * (1 + eps)) | ((e == hi) & (lo == hi))
        else:
            surely = keep
        slack = e[keep & ~surely].sum() + eps * e.sum()
        before, mass = e[:tok[r]][surely[:tok[r]]].sum(), e[surely].sum()
        assert u[r] * mass >= before - slack and u[r] * mass <= before + e[tok[r]] + slack
        assert abs(lp[r] - np.log(e[tok[r]] / mass)) <= 2e-5 + 2 * slack / mass
    again = Cc.sample_top_p(x.clone(), 11, ids, 3, T, top_p, None)
    assert np.array_equal(again[0].cpu().numpy(), tok) and np.array_equal(again[1].cpu().numpy(), lp)


def test_rows_without_mass_give_a_valid_token():
    from ferrl_b200.ops import cuda as Cc
    x = torch.full((3, 20000), float("-inf"), device="cuda", dtype=torch.bfloat16)
    x[1, 777] = float("inf")
    x[2] = float("nan")
    tok, lp = Cc.sample_top_p(x, 1, torch.arange(3, device="cuda"), 0, 1.0, 0.9, None)
    assert tok.tolist() == [0, 777, 0] and bool((lp <= 0).all())


def _us(x, top_p, T=1.0):
    from ferrl_b200.ops import cuda as Cc
    ids, flush, ts = torch.arange(x.shape[0], device="cuda"), torch.empty(64 << 20, device="cuda"), []
    for _ in range(15):
        flush.zero_()                                                         # the rows come from HBM
        a, b = torch.cuda.Event(True), torch.cuda.Event(True)
        a.record()
        Cc.sample_top_p(x, 7, ids, 3, T, top_p, None)
        b.record()
        torch.cuda.synchronize()
        ts.append(a.elapsed_time(b) * 1e3)
    return sorted(ts)[7]


def _plain(rows, V, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows)
    return (torch.randn(rows, V, generator=g, device="cuda") * 2.5).to(dtype)


@pytest.mark.no_canary
@pytest.mark.parametrize("rows,V", [(128, 151936), (512, 50264)])
def test_rows_without_a_cut_cost_less(rows, V):
    """The sum of the masses is all that they want: 53 us before rows were counted, 71 with the counts, at 128 x 151936."""
    x = _plain(rows, V, torch.bfloat16)
    assert _us(x, None) < 0.75 * _us(x, 0.95)


@pytest.mark.no_canary
@pytest.mark.parametrize("kind", ["masked", "flat"])
def test_32_bit_rows_of_one_key_or_with_finite_masks_cost_no_more(kind):
    """Entries without a mass and segments of one key need no narrowing (128 x 151936: 311 and 419 us with it, 166 a plain row)."""
    x = _plain(128, 151936, torch.float32)
    plain = _us(x, 0.95)
    x = x * 0 if kind == "flat" else x.index_fill(1, torch.arange(0, 151936, 2, device="cuda"), -1e4)
    assert _us(x, 0.95) < 1.15 * plain


def _kind(kind, rows, V):
    """-> (bf16 logits, top-p, temperature) of rows whose values are not spread over a few octaves about one."""
    x, even = _plain(rows, V, torch.float32), torch.arange(0, V, 2, device="cuda")
    x, top_p, T = {"few masked": lambda: (x.index_fill(1, even[3:25], -1e4), 0.95, 1.0), "half masked": lambda: (x.index_fill(1, even, -1e4), 0.95, 1.0),
                   "masked by the least value": lambda: (x.index_fill(1, even, torch.finfo(torch.bfloat16).min), 0.95, 1.0),
                   "far up": lambda: (x + 600, 0.95, 1.0), "wide": lambda: (x * 120, 0.95, 1.0), "wide and hot": lambda: (x * 120, 0.95, 100.0),
                   "nearly flat": lambda: (x * 4e-5, 0.95, 1.0), "cut about zero": lambda: (x * (1.645 / 2.5), 0.95, 1.0),
                   "half zero": lambda: (x.index_fill(1, even, 0.0), 0.95, 1.0), "rectified": lambda: (x.clamp_min(0), 0.9, 1.0),
                   "all zero": lambda: (torch.zeros_like(x), 0.5, 1.0), "one peak": lambda: (x.index_fill(1, even[7:8], 300.0), 0.95, 1.0),
                   "two scales": lambda: ((x * 0.8 - 3).index_fill(1, even, 0.0) + (x * 8e-5).index_fill(1, torch.arange(1, V, 2, device="cuda"), 0.0), 0.7, 1.0),
                   "tail below": lambda: (x.index_fill(1, even[4:8], -2000.0), 0.99999, 1000.0),
                   "large outliers, hot": lambda: (x.index_fill(1, even[100:160], 5e4).index_fill(1, even[200:260], -5e4), 0.3, 1e5),
                   "small cut, hot": lambda: (x.index_fill(1, even[100:160], 3e-6).index_fill(1, even[200:900], -3e-6), 0.5, 50.0)}[kind]()
    return x.bfloat16(), top_p, T


KINDS = ["few masked", "half masked", "masked by the least value", "far up", "wide", "wide and hot", "nearly flat", "cut about zero", "half zero",
         "rectified", "all zero", "one peak", "two scales", "tail below", "large outliers, hot", "small cut, hot"]


@pytest.mark.parametrize("rows,V", [(3, 20000), (40, 50257), (2, 262144)])
@pytest.mark.parametrize("kind", KINDS)
def test_16_bit_rows_draw_what_the_same_values_draw_in_32(kind, rows, V):
    """The two paths share no counter, list or segment; the masses are the same integers.  Where neighbouring 16-bit values have one
    32-bit probability (nearly flat rows) the 32-bit cut keeps both, so the log-prob moves by their share of the kept mass."""
    from ferrl_b200.ops import cuda as Cc
    x, top_p, T = _kind(kind, rows, V)
    for seed in (1, 2, 3):
        a, b = (Cc.sample_top_p(t, seed, torch.arange(rows, device="cuda"), 3, T, top_p, None) for t in (x, x.float()))
        if kind in ("nearly flat", "cut about zero", "small cut, hot", "wide and hot", "large outliers, hot", "two scales"):
            assert float((a[1] - b[1]).abs().max()) < 0.02
        else:
            assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


@pytest.mark.no_canary
@pytest.mark.parametrize("rows,V", [(128, 151936), (512, 50264)])
def test_values_outside_the_usual_octaves_cost_no_more(rows, V):
    """Finite masks, large, small and repeated values are counted, skipped or listed.  128 x 151936, us: without that 120 to 180 as one
    CTA a row, and 240 to 470 by the general path."""
    plain = _us(_plain(rows, V, torch.bfloat16), 0.95)
    slow = {k: _us(*_kind(k, rows, V)) / plain for k in KINDS if k != "large outliers, hot"}
    assert all(r < (3.5 if k == "two scales" else 1.9 if k in ("half zero", "rectified", "all zero") else 1.4) for k, r in slow.items()), slow


def test_many_rows_of_a_vast_vocabulary():
    """One CTA a row would add more than 2^21 masses into a 32-bit histogram; alone, a row is shared by a whole cluster."""
    from ferrl_b200.ops import cuda as Cc
    rows, V = 384, 4300000
    low = -13.9 - 0.001 * torch.arange(rows, device="cuda").float()[:, None]
    x = low.expand(rows, V).contiguous()
    x[:, ::2] -= 1e-4                                         # two keys of one segment
    x[:, 7] = 0
    ids = torch.arange(rows, device="cuda")
    tok, lp = Cc.sample_top_p(x, 5, ids, 1, 1.0, 0.9, None)
    for r in range(0, rows, 24):
        t, l = Cc.sample_top_p(x[r:r + 1], 5, ids[r:r + 1], 1, 1.0, 0.9, None)
        assert int(t) == int(tok[r]) and float(l) == float(lp[r])
