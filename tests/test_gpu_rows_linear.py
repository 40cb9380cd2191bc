"""The tensor-core linear kernel at the edges of its tiles, and the packed step where its row tiles change size."""
import numpy as np
import pytest

import orc
import rwkv_rsv_b200 as rsv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 5, 16, 17, 63, 64, 65, 129])
@pytest.mark.parametrize("m,k,int8", [(128, 128, True), (384, 2560, True), (2560, 1024, True), (96, 512, False), (130, 96, False), (2560, 2560, False)])
def test_linear_tile_edges(rows, m, k, int8):
    rng = np.random.default_rng(rows * 1000 + m + k)
    x = (rng.standard_normal((rows, k)) * np.exp(rng.uniform(-4, 4, (rows, 1)))).astype(np.float32)
    if int8:
        idx = rng.integers(0, 256, size=(m, k), dtype=np.uint8)
        scale = (rng.random((m, 1)) * 0.01 + 0.001).astype(np.float16)
        zero = (-128.0 * scale.astype(np.float32)).astype(np.float16)
        sz = np.ascontiguousarray(np.repeat((zero.view(np.uint16).astype(np.uint32) << 16) | scale.view(np.uint16).astype(np.uint32), k // 128, axis=1))
        got, w = rsv.op_linear(x, idx, sz, path=1), orc.dequant_int8(idx, sz).astype(np.float64)
    else:
        wh = (rng.standard_normal((m, k)) * 0.02).astype(np.float16)
        got, w = rsv.op_linear(x, wh, None, path=1), wh.astype(np.float64)
    want = x.astype(np.float64) @ w.T
    amax, absw, absxw = np.abs(x).max(1, keepdims=True).astype(np.float64), np.abs(w).sum(1)[None, :], np.abs(x).astype(np.float64) @ np.abs(w).T
    if int8:  # the only error: each activation to half a step of 2^-27 of its row's power-of-two scale (at most twice the maximum); then one rounding
        bound = 2.0 ** -27 * amax * absw + 2.0 ** -23 * np.abs(want)
    else:  # hi + lo halves carry 21 bits of the scaled activation, the tensor core adds k products in fp32
        bound = 2.0 ** -21 * 2 * amax * absw + k * 2.0 ** -24 * absxw
    assert np.all(np.abs(got - want) <= bound + 1e-30), float((np.abs(got - want) / bound).max())


# enough tiles that K is not split and two CTAs share a tile of 256 weight rows: full and ragged row tiles, an odd number of 128-row
# weight tiles, the last of them partly or wholly past the end
@pytest.mark.parametrize("rows,m,k,int8", [(513, 2560, 1024, True), (640, 2688, 384, True), (513, 2560, 704, False), (577, 2570, 640, False)])
def test_linear_tiles_of_a_cta_pair(rows, m, k, int8):
    test_linear_tile_edges(rows, m, k, int8)


@pytest.mark.parametrize("name", ["fp16", "int8", "int8g"])
def test_step_sizes_agree_with_the_cpu_path(tiny_paths, name):
    # 16 / 17: operands built inside or outside the GEMM; 32 / 33, 64 / 65: one or two row tiles (per-group and other weights)
    b, o = rsv.ModelBuilder(tiny_paths[name]).build(), orc.OracleModel(tiny_paths[name])
    rng = np.random.default_rng(3)
    for n in (2, 16, 17, 32, 33, 64, 65, 150):
        toks = rng.integers(0, b.info().num_vocab, size=n).astype(np.uint32)
        b.reset()
        o.reset()
        lg, want = b.infer_seq(toks), o.forward(toks)
        # fp32 through the layers in another summation order: a few ulps of the logits' scale per layer
        assert float(np.sqrt(np.mean((lg - want) ** 2))) <= 64 * 2.0 ** -24 * max(1.0, float(np.abs(want).max())), n
        assert np.abs(b.state_back() - o.state_back()).max() <= 1e-4 * max(1.0, float(np.abs(o.state_back()).max()))


# fp16 tiles of up to 108 rows share an SM when K is split, larger ones have it to themselves; m = 2048: few tiles, which are split; 9600: as many
# tiles as a launch of one CTA per SM holds, which are not; 704: a tile of fewer than 16 K blocks, which no persistent CTA takes
@pytest.mark.parametrize("rows", [210, 216, 217, 256])
@pytest.mark.parametrize("m,k", [(2048, 2560), (9600, 1536), (9600, 704)])
def test_linear_fp16_tiles_that_need_a_whole_sm(rows, m, k):
    test_linear_tile_edges(rows, m, k, False)
