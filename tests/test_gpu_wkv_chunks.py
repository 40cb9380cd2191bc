"""WKV-7 sixteen tokens at a time: ragged last chunks, several segments, decays at both ends of a model's range, against the recurrence in
64 bits.  The kernels run where the automatic choice takes them: segments of 160 tokens and more, at most an SM for each of a head's two halves."""
import numpy as np
import pytest

import rwkv_rsv_b200 as rsv

pytestmark = pytest.mark.gpu


def _case(nseg, T, H, seed, gate, decays):
    rng = np.random.default_rng(seed)
    C = H * 64
    n = lambda *s: rng.standard_normal(s).astype(np.float32)  # noqa: E731
    u = lambda *s: rng.random(s).astype(np.float32)  # noqa: E731
    d = dict(r=n(nseg, T, C), k=n(nseg, T, C), v=n(nseg, T, C), w=(decays[0] + (decays[1] - decays[0]) * u(nseg, T, C)).astype(np.float32), a=u(nseg, T, C), g=n(nseg, T, C),
             k_k=n(C), k_a=u(C), r_k=0.1 * n(C), lnx_w=1 + 0.1 * n(C), lnx_b=0.1 * n(C), state=0.1 * n(nseg, H, 64, 64))
    d = {k: v.astype(np.float32) for k, v in d.items()}
    if gate:
        d.update(vgate=u(nseg, T, C), vfirst=n(nseg, T, C))
    return d


def _exact(d):
    """y and state of every segment in 64 bits."""
    x = {k: v.astype(np.float64) for k, v in d.items()}
    nseg, T, C = x["r"].shape
    H = C // 64
    hd = lambda m: m.reshape(m.shape[:-1] + (H, 64))  # noqa: E731
    v = x["v"] + x["vgate"] * (x["vfirst"] - x["v"]) if "vgate" in x else x["v"]
    kk = hd(x["k"] * x["k_k"])
    kk = kk / np.maximum(np.sqrt((kk ** 2).sum(-1, keepdims=True)), 1e-12)
    kt = x["k"] + x["k_a"] * (x["k"] * x["a"] - x["k"])
    b, r, w, k, v, g = -kk * hd(x["a"]), hd(x["r"]), hd(x["w"]), hd(kt), hd(v), hd(x["g"])
    S, out = x["state"].copy(), np.empty_like(r)
    for t in range(T):
        sa = np.einsum("nhij,nhj->nhi", S, kk[:, t])
        S = S * w[:, t, :, None, :] + sa[..., None] * b[:, t, :, None, :] + v[:, t, :, :, None] * k[:, t, :, None, :]
        y = np.einsum("nhij,nhj->nhi", S, r[:, t])
        y = (y - y.mean(-1, keepdims=True)) / np.sqrt(y.var(-1, keepdims=True) + 64e-5)
        y = y * hd(x["lnx_w"]) + hd(x["lnx_b"]) + (r[:, t] * k[:, t] * hd(x["r_k"])).sum(-1, keepdims=True) * v[:, t]
        out[:, t] = y * g[:, t]
    return out.reshape(nseg, T, C), S


@pytest.mark.parametrize("nseg,T,H,gate,decays", [(1, 160, 8, False, (0.5453, 1.0)), (9, 161, 8, True, (0.5453, 1.0)), (2, 175, 37, True, (0.999, 1.0)), (1, 320, 40, True, (0.5453, 1.0)), (1, 321, 8, False, (0.5453, 0.5454)), (9, 335, 8, True, (0.5453, 1.0)), (1, 512, 3, True, (0.999, 1.0)),
                                                  (2, 387, 37, False, (0.5453, 1.0))])
def test_chunks_match_the_recurrence_in_64_bits(nseg, T, H, gate, decays):
    d = _case(nseg, T, H, 7 * T + H, gate, decays)
    y, s = rsv.op_wkv7(variant=0, **d)
    yw, sw = _exact(d)
    # in fp32 a state that decays is off by about two roundings (2^-24 each) in the 2-norm, one that does not by three (the chunks round it once each); twice
    # that, and four times that for the largest
    assert np.linalg.norm(s - sw) <= 2.0 ** -24 * 6 * np.linalg.norm(sw) and np.abs(s - sw).max() <= 2.0 ** -22 * 6 * np.abs(sw).max()
    assert np.linalg.norm(y - yw) <= 2.0 ** -24 * 6 * np.linalg.norm(yw) and np.abs(y - yw).max() <= 2.0 ** -22 * 6 * np.abs(yw).max()


# No further from 64 bits than the token-by-token kernel on the same inputs (two hundredths of room: the errors are sums over 1e5 roundings)
@pytest.mark.parametrize("decays", [(0.5453, 0.5454), (0.5453, 1.0), (0.7, 0.8), (0.9, 1.0), (0.999, 1.0)])
def test_chunks_are_as_precise_as_token_by_token(decays):
    off = np.zeros((2, 2))
    for seed, T in ((1, 160), (2, 505)):
        d = _case(1, T, 8, seed, True, decays)
        want = _exact(d)
        for i, variant in enumerate((0, 3)):
            off[i] += [float(np.sum((g - w) ** 2) / np.sum(w ** 2)) for g, w in zip(rsv.op_wkv7(variant=variant, **d), want)]
    assert (np.sqrt(off[0]) <= 1.02 * np.sqrt(off[1])).all(), np.sqrt(off)


def test_other_decays_go_token_by_token():
    # zero decays have no running products to divide by
    d = _case(1, 400, 8, 5, True, (0.0, 1.0))
    d["w"][0, 40] = 0.0
    y, s = rsv.op_wkv7(variant=0, **d)
    ref, sref = rsv.op_wkv7(variant=3, **d)
    assert np.array_equal(y, ref) and np.array_equal(s, sref) and np.isfinite(s).all()


# The scratch of a prompt's chunks grows with the prompt: lengths up and down, against the same prompts in steps that are too short for the matrix form
def test_prompts_of_growing_length(tmp_path):
    b = rsv.ModelBuilder(rsv.write_synthetic(str(tmp_path / "m.st"), "tiny", seed=3)).build()
    for n in (160, 176, 320, 400, 512, 170, 511):
        toks = np.random.default_rng(n).integers(0, 4096, size=n).astype(np.uint32)
        b.reset()
        lg = b.infer_chunked(toks, 512)
        b.reset()
        want = b.infer_chunked(toks, 128)
        # fp32 through the layers in another summation order: a few ulps of the logits' scale per layer
        assert float(np.sqrt(np.mean((lg - want) ** 2))) <= 64 * 2.0 ** -24 * max(1.0, float(np.abs(want).max())), n
    b.state.close()
    b.model.close()
