"""What the sampler does with masked tokens (-inf, the lowest float), in rows of one CTA, of a cluster and of the kernel for large vocabularies."""
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


def test_unmix_is_the_inverse():
    for z in (0, 1, 12345, 0x80000000, 0xFFFFFFFF):
        assert f32(orc.lib().orc_u01(_unmix(z))) == f32(f32(z) / f32(4294967296.0))


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
