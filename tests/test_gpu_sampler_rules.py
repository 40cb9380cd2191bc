"""What the sampler promises whatever the rounding: a drawn token is one that top-k and top-p kept, and masked tokens (-inf, the lowest
float) are never drawn beside others.  Rows of one CTA, of a cluster and of the kernel for large vocabularies."""
import numpy as np
import pytest

import orc
import rwkv_rsv_b200 as rsv

pytestmark = pytest.mark.gpu

f32 = np.float32


def _unmix(z):
    """The seed whose draw is u = float(z) / 2^32 (the sampler's integer mix, backwards: every step of it is a bijection of 32 bits)."""
    m = 0xFFFFFFFF
    z ^= z >> 16
    z = z * pow(0xC2B2AE35, -1, 1 << 32) & m
    z ^= z >> 13 ^ z >> 26
    z = z * pow(0x85EBCA6B, -1, 1 << 32) & m
    z ^= z >> 16
    return (z - 0x9E3779B9) & m


def _running_sums(p, ctas, threads, per):
    """The kernels' fp32 prefix sums: start and end of every thread's range of `per` tokens, and the total."""
    e = np.zeros(ctas * threads * per, f32)
    e[:p.size] = p
    e = e.reshape(ctas, threads // 32, 32, per)
    csum = np.zeros(e.shape[:3], f32)
    for q in range(per):
        csum = csum + e[..., q]
    incl = csum.copy()
    for o in (1, 2, 4, 8, 16):
        up = np.zeros_like(incl)
        up[..., o:] = incl[..., :-o]
        incl = np.where(np.arange(32) >= o, incl + up, incl)
    warps = incl[..., 31]
    wbase = np.zeros(warps.shape, f32)
    for i in range(1, warps.shape[1]):
        wbase[:, i] = wbase[:, i - 1] + warps[:, i - 1]
    kept = wbase[:, -1] + warps[:, -1]
    base = np.zeros(ctas, f32)
    for c in range(1, ctas):
        base[c] = base[c - 1] + kept[c - 1]
    total = base[-1] + kept[-1]
    start = ((base[:, None] + wbase)[..., None] + incl) - csum
    end = start
    for q in range(per):
        end = end + e[..., q]
    return start.ravel(), end.ravel(), csum.ravel() > 0, total


def _seeds_between_steps(p, ctas, threads, per):
    """Seeds whose u lies in a gap: at or above what every kept thread before it reached, below where a thread without kept tokens starts."""
    start, end, has, total = _running_sums(p, ctas, threads, per)
    seeds = []
    reach = np.maximum.accumulate(np.where(has, end, f32(0)))
    for t in np.nonzero(~has & (start > reach))[0]:
        f = f32(reach[t] / total)
        for _ in range(8):
            f = np.nextafter(f, f32(0))
        for _ in range(16):
            if reach[t] <= f32(f * total) < start[t]:
                z = int(np.float64(f) * 2 ** 32)
                if z < 2 ** 32 and f32(z) == f32(np.float64(f) * 2 ** 32):
                    seeds.append(_unmix(z))
                    break
            f = np.nextafter(f, f32(2))
    return seeds


def test_unmix_is_the_inverse():
    for z in (0, 1, 12345, 0x80000000, 0xFFFFFFFF):
        assert f32(orc.lib().orc_u01(_unmix(z))) == f32(f32(z) / f32(4294967296.0))


# a row of one cluster of CTAs (8192 logits each), of one CTA of a cluster kernel, and of the kernel for larger vocabularies
@pytest.mark.parametrize("v,ctas,threads,per", [(65536, 8, 512, 16), (8192, 1, 512, 16), (70000, 1, 1024, 69)])
def test_drawn_tokens_were_kept(v, ctas, threads, per):
    rng = np.random.default_rng(v)
    logits, rows = [], []
    for n in range(20, 400):
        # n equally probable tokens; everything else is cut by top-k
        lg = np.full(v, -100.0, f32)
        lg[rng.choice(v - 1, n, replace=False)] = 0.0  # the last token is never kept
        p = np.where(lg == 0, f32(1) / f32(n), f32(0)).astype(f32)
        seeds = _seeds_between_steps(p, ctas, threads, per)[:2] + [_unmix(0xFFFFFFFF), _unmix(0)]  # and u = 1 and 0
        for s in seeds:
            logits.append(lg)
            rows.append(orc.pack_sampler(seed=s, top_k=n, top_p=1.0))
        if len(rows) >= 200:
            break
    logits = np.stack(logits)
    got = rsv.op_sample(logits, np.stack(rows)).astype(np.int64)
    bad = [(i, int(t)) for i, t in enumerate(got) if logits[i, t] != 0]
    assert not bad, bad[:5]


def test_drawn_tokens_of_a_nucleus_were_kept():
    v, n = 16384, 1500
    lg = (np.random.default_rng(5).standard_normal(v) * 4).astype(f32)
    logits = np.broadcast_to(lg, (n, v))
    got = rsv.op_sample(logits, np.stack([orc.pack_sampler(seed=s, top_p=0.7) for s in range(n)]))
    p = np.sort(np.exp(np.float64(lg) - lg.max()) / np.exp(np.float64(lg) - lg.max()).sum())[::-1]
    k = int(np.searchsorted(np.cumsum(p), 0.7)) + 2  # (one more: the kernel's fp32 sum may need another pick)
    assert lg[got].min() >= np.sort(lg)[::-1][k]


# Every logit below the sampler's floor: such tokens count as -1e30 and are then equally probable.  V = 5000 and 65536 are rows of a cluster,
# 70000 of the kernel for larger vocabularies; u is kept away from the steps of the sum.
@pytest.mark.parametrize("v", [5000, 65536, 70000])
@pytest.mark.parametrize("value", [-np.inf, -3.4028235e38])
@pytest.mark.parametrize("k,top_p", [(0, 1.0), (40, 1.0), (3000, 1.0)])
def test_fully_masked_rows_are_drawn_uniformly(v, value, k, top_p):
    u = np.array([0.031, 0.27, 0.5, 0.77, 0.93])
    rows = np.stack([orc.pack_sampler(seed=_unmix(int((np.floor(x * v) + 0.5) / v * 2 ** 32)), top_k=k, top_p=top_p) for x in u])
    got = rsv.op_sample(np.full((u.size, v), value, f32), rows)
    assert np.abs(got.astype(np.float64) - np.floor(u * v)).max() <= 1 + v * 2.0 ** -17  # at most 106 additions deep (69 + 5 + 32), 2^-24 each


# masked tokens beside real ones are never drawn, also when fewer are left than top-k asks for
@pytest.mark.parametrize("v", [5000, 65536, 70000])
@pytest.mark.parametrize("k,top_p", [(0, 1.0), (50, 0.9), (0, 0.9), (600, 0.9)])
def test_masked_tokens_are_not_drawn(v, k, top_p):
    rng = np.random.default_rng(v + k)
    lg = np.full((64, v), -np.inf, f32)
    allowed = rng.choice(v, 30, replace=False)
    lg[:, allowed] = (rng.standard_normal((64, 30)) * 2).astype(f32)
    rows = np.stack([orc.pack_sampler(seed=s, top_k=k, top_p=top_p, temperature=0.8) for s in range(64)])
    got = rsv.op_sample(lg, rows)
    assert set(int(g) for g in got) <= set(int(a) for a in allowed)
    assert [int(g) for g in got[:8]] == [orc.sample(lg[s], seed=s, top_k=k, top_p=top_p, temperature=0.8) for s in range(8)]


@pytest.mark.parametrize("v", [5000, 65536, 70000])
def test_rows_with_a_nan_or_an_infinity(v):
    # no sum of such a row exceeds u, so the answer is the last token, as on the CPU path
    lg = np.random.default_rng(v).standard_normal((2, v)).astype(f32)
    lg[0, 100], lg[1, 100] = np.nan, np.inf
    got = rsv.op_sample(lg, np.stack([orc.pack_sampler(seed=s) for s in (1, 2)]))
    assert [int(g) for g in got] == [v - 1, v - 1] == [orc.sample(lg[s], seed=s + 1) for s in range(2)]


# The top-p walk takes eight entries of the sorted list at a time until their sum reaches top_p: the last kept token at the ends of such a group, the list's
# own end (512), and lists of one warp's and of several warps' entries
@pytest.mark.parametrize("kept,top_k", [(1, 0), (7, 0), (8, 0), (9, 0), (16, 0), (17, 0), (65, 0), (512, 0), (8, 8), (13, 13), (9, 40), (33, 50), (700, 0)])
def test_top_p_keeps_exactly_the_largest_that_reach_it(kept, top_k):
    rng = np.random.default_rng(kept)
    V, n = 4096, min(kept, 512)  # (at most 512 picks)
    rows = 400 if kept <= 33 else 24 * n  # the least likely of n kept tokens goes undrawn in 24 n draws with probability e^-18
    order = rng.permutation(V)
    logits = np.empty(V, np.float32)
    logits[order] = -1e-3 * np.arange(V, dtype=np.float32)  # nearly flat: every kept token is drawn sooner or later
    p = np.exp(logits[order].astype(np.float64))
    if top_k:
        p[top_k:] = 0.0
    p /= p.sum()
    top_p = float(min(0.999999, p[:kept].sum() - 0.5 * p[kept - 1]))
    got = rsv.op_sample(np.repeat(logits[None], rows, 0), np.stack([orc.pack_sampler(seed=77 * r + 1, top_p=top_p, top_k=top_k) for r in range(rows)])).astype(np.int64)
    rank = np.empty(V, np.int64)
    rank[order] = np.arange(V)
    assert set(rank[got].tolist()) == set(range(n))
