"""The single-session decode kernel at the widths where its division of K and of the heads' rank vectors changes, and the sampler's
cluster at the sizes where its number of CTAs and its way to the k-th largest change."""
import os

import numpy as np
import pytest

import orc
import rwkv_rsv_b200 as rsv

pytestmark = pytest.mark.gpu


# 768: 48 channels per warp (a warp's last 32 are half empty), ranks that are no whole step of 16; 1024 and 1536: an instantiation's full
# and partial width; 2560 per group: groups of 128 that straddle two warps; 1536 also has a quantised head
@pytest.mark.parametrize("n_embd,quant,quant_head,ranks", [(768, 0, False, (24, 40, 8, 72)), (1024, 1, False, (32, 32, 32, 32)), (1536, 1, True, (64, 64, 32, 128)),
                                                          (2560, 2, False, (96, 96, 64, 320))])
def test_decode_kernel_widths(tmp_path, n_embd, quant, quant_head, ranks):
    p = rsv.write_synthetic(os.path.join(str(tmp_path), "m.st"), "tiny", seed=0, quant=quant, quant_head=quant_head, n_layer=2, n_embd=n_embd, n_head=n_embd // 64,
                            ffn_hidden=4 * n_embd, vocab=1000, w_mid=ranks[0], a_mid=ranks[1], v_mid=ranks[2], g_mid=ranks[3])
    b, o = rsv.ModelBuilder(p).build(), orc.OracleModel(p)
    toks = np.random.default_rng(5).integers(0, 1000, size=9).astype(np.uint32)
    for n in (1, 9):  # 9: the tokens of one launch follow each other through the exchange buffers
        b.reset()
        o.reset()
        lg, want = b.infer_tokens(toks[:n]), o.forward(toks[:n])
        # fp32 through the layers in another summation order: a few ulps of the logits' scale per layer
        assert float(np.sqrt(np.mean((lg - want) ** 2))) <= 64 * 2.0 ** -24 * max(1.0, float(np.abs(want).max())), n
        assert np.abs(b.state_back() - o.state_back()).max() <= 1e-4 * max(1.0, float(np.abs(o.state_back()).max()))
    b.state.close()
    b.model.close()


# 8192 / 8193: one CTA or two; 65536: all eight; k = 512 / 513: the sorted list serves top-p or not; k = 3000: more candidates than the
# list holds, so the k-th largest comes from the radix passes
@pytest.mark.parametrize("v", [1, 7, 8192, 8193, 65536])
@pytest.mark.parametrize("k,top_p", [(0, 0.9), (1, 1.0), (50, 0.9), (512, 0.9), (513, 0.9), (3000, 1.0)])
def test_sampler_cluster_sizes(v, k, top_p):
    lg = (np.random.default_rng(v + k).standard_normal((3, v)) * 3).astype(np.float32)
    lg[2] = np.round(lg[2])  # ties
    rows = np.stack([orc.pack_sampler(seed=9 + r, top_k=k, top_p=top_p) for r in range(3)])
    got = rsv.op_sample(lg, rows)
    want = [orc.sample(lg[r], seed=9 + r, top_k=k, top_p=top_p) for r in range(3)]
    assert [int(g) for g in got] == [int(x) for x in want]
