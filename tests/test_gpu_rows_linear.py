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


# several row tiles of few K blocks, a CTA or (the first fp16 shape) a pair that splits K per tile: full and ragged row tiles, an odd number of weight
# tiles, a partial last one
@pytest.mark.parametrize("rows,m,k,int8", [(513, 2560, 1024, True), (640, 2688, 384, True), (513, 2560, 704, False), (577, 2570, 640, False)])
def test_linear_several_row_tiles(rows, m, k, int8):
    test_linear_tile_edges(rows, m, k, int8)


# The persistent kernel: several row tiles, more tiles than SMs (so that K is not split), 16 K blocks and more, int8 or fp16 tiles of more than 64
# rows.  129: three tiles of 43 rows (no multiple of 4); 201: the last tile is one row shorter; 4033: the last tile is a single row; 10250
# and 9640 weight rows: a partial last weight tile; 257, 513 and 1025 rows of fp16: ragged last tiles of 85, 101 and 113 rows
@pytest.mark.parametrize("rows,m,k,int8", [(129, 10240, 2560, True), (201, 10240, 2560, True), (4033, 384, 2048, True), (257, 10250, 1088, False), (513, 10250, 1088, False),
                                           (1025, 9640, 1024, False)])
def test_linear_persistent_tiles(rows, m, k, int8):
    test_linear_tile_edges(rows, m, k, int8)


# ... and tiles of few K blocks once there are four turns of them: a ragged last row tile (1025 rows are 17 tiles of 61, 1024 of fp16 weights eight of 128), a partial last weight tile
@pytest.mark.parametrize("rows,m,k,int8", [(1025, 5120, 512, True), (1025, 9610, 320, False), (1024, 9600, 64, False)])
def test_linear_persistent_short_rows(rows, m, k, int8):
    test_linear_tile_edges(rows, m, k, int8)


# ... with (scale, zero) pairs that are not symmetric around code 128 in every row, in one row of a tile, or with codes and activations at their limits (the integer
# sums reach 2^47)
@pytest.mark.parametrize("kind", ["asymmetric", "one row", "limits"])
def test_linear_persistent_zero_points(kind):
    rows, m, k = 513, 2560, 10240 if kind == "limits" else 2560
    rng = np.random.default_rng(len(kind))
    x = np.ones((rows, k), np.float32) if kind == "limits" else rng.standard_normal((rows, k)).astype(np.float32)
    idx = rng.integers(0, 2, size=(m, 1), dtype=np.uint8) * np.full((1, k), 255, np.uint8) if kind == "limits" else rng.integers(0, 256, size=(m, k), dtype=np.uint8)
    scale = (rng.random((m, 1)) * 0.01 + 0.001).astype(np.float16)
    zero = (-128.0 * scale.astype(np.float32)).astype(np.float16)
    if kind == "asymmetric":
        zero = (rng.standard_normal((m, 1)) * 0.3).astype(np.float16)
    elif kind == "one row":
        zero[200] = 0.25
    sz = np.ascontiguousarray(np.repeat((zero.view(np.uint16).astype(np.uint32) << 16) | scale.view(np.uint16).astype(np.uint32), k // 128, axis=1))
    got, w = rsv.op_linear(x, idx, sz, path=1), orc.dequant_int8(idx, sz).astype(np.float64)
    want = x.astype(np.float64) @ w.T
    bound = 2.0 ** -27 * np.abs(x).max(1, keepdims=True) * np.abs(w).sum(1)[None, :] + 2.0 ** -23 * np.abs(want)  # (as above)
    assert np.all(np.abs(got - want) <= bound + 1e-30), float((np.abs(got - want) / bound).max())


def _int8_words(scale, zero, groups):
    word = (zero.view(np.uint16).astype(np.uint32) << 16) | scale.view(np.uint16).astype(np.uint32)
    return np.ascontiguousarray(np.repeat(word[:, None], groups, axis=1))


# An int8 output is the exact sum, rounded once, whichever kernel takes its row (2 and 16 rows: split along K where K is long; 513: the persistent one).  The activations are whole
# numbers of at most 20 bits times a power of two, so that their fixed-point values are exact, and the products with the scales fit fp64.
@pytest.mark.parametrize("kind", ["ordinary", "small sums", "limits", "asymmetric", "one row"])
@pytest.mark.parametrize("rows", [2, 16, 513])
def test_int8_sums_are_rounded_once(rows, kind):
    m, k = 2560, 10240 if kind == "limits" else 2560
    rng = np.random.default_rng(rows + len(kind))
    x = rng.integers(-(1 << 20), 1 << 20, size=(rows, k)).astype(np.float64)
    idx = rng.integers(0, 256, size=(m, k), dtype=np.uint8)
    if kind == "small sums":  # a large activation against the code of zero, and a few of the smallest: sums of both signs down to one step of the fixed point
        x = np.where(rng.random((rows, k)) < 4 / k, rng.integers(-3, 4, size=(rows, k)), 0).astype(np.float64)
        x[:, 0] = 1 << 26
        idx[:, 0] = 128
    elif kind == "limits":
        x = np.where(rng.random((rows, 1)) < 0.5, 1.0, -1.0) * ((1 << 20) - rng.integers(0, 9, size=(rows, k)))
        idx = (255 * rng.integers(0, 2, size=(m, 1)) + np.zeros((1, k))).astype(np.uint8)
    scale = (rng.integers(1024, 2048, size=m) * 2.0 ** -14).astype(np.float16)  # 11 bits
    scale[:4] = [0.0, 2.0 ** -24, -0.0078125, 511.0] if kind in ("ordinary", "small sums") else scale[:4]
    zero = (-128.0 * scale.astype(np.float32)).astype(np.float16)
    if kind == "asymmetric":
        # zero points of under a step of the codes, of 100 to 155 steps, and of up to 1000
        zero = np.choose(np.arange(m) % 3, [rng.integers(-2048, 2048, size=m) * 2.0 ** -14, -rng.uniform(100, 155, size=m) * scale, rng.uniform(-60, 60, size=m)]).astype(np.float16)
    elif kind == "one row":
        zero[200] = 0.25
    got = rsv.op_linear((x * 2.0 ** -9).astype(np.float32), idx, _int8_words(scale, zero, k // 128), path=1)
    q, t = x @ idx.astype(np.float64).T, x.sum(1)[:, None]  # (whole numbers under 2^43)
    want = (q * scale.astype(np.float64) + t * zero.astype(np.float64)) * 2.0 ** -9
    assert np.array_equal(got, want.astype(np.float32)), (int((got != want.astype(np.float32)).sum()), float(np.abs(got / np.where(want == 0, 1, want) - 1).max()))


# The same kernel as a step uses it: int8 next to fp16 problems in one launch, rank projections that are partial weight tiles, the maxima of
# ffn.key's outputs (8200: its last weight tile has eight rows), row tiles of 44, 51, 65 and 86 rows
@pytest.mark.parametrize("quant,ffn", [(1, 8192), (0, 8200)])
def test_step_of_persistent_tiles_agrees_with_the_cpu_path(tmp_path, quant, ffn):
    p = rsv.write_synthetic(str(tmp_path / "m.st"), "tiny", seed=0, quant=quant, n_layer=1, n_embd=2048, n_head=32, ffn_hidden=ffn, vocab=300, w_mid=24, a_mid=40,
                            v_mid=8, g_mid=72)
    b, o = rsv.ModelBuilder(p).build(), orc.OracleModel(p)
    for n in (130, 201, 257):
        toks = np.random.default_rng(n).integers(0, 300, size=n).astype(np.uint32)
        b.reset()
        o.reset()
        lg, want = b.infer_seq(toks), o.forward(toks)
        # fp32 through the layer in another summation order: a few ulps of the logits' scale
        assert float(np.sqrt(np.mean((lg - want) ** 2))) <= 64 * 2.0 ** -24 * max(1.0, float(np.abs(want).max())), n
        assert np.abs(b.state_back() - o.state_back()).max() <= 1e-4 * max(1.0, float(np.abs(o.state_back()).max()))
    b.state.close()
    b.model.close()


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


# One row tile and more weight tiles than two CTAs per SM hold (a vocabulary head): the persistent kernel with a single row tile; 38016 and 38100: 297
# and 298 weight tiles, the last of 84 rows
@pytest.mark.parametrize("rows,m,k,int8", [(1, 38016, 1024, False), (3, 38100, 1088, False), (64, 38016, 2048, True)])
def test_linear_persistent_with_one_row_tile(rows, m, k, int8):
    test_linear_tile_edges(rows, m, k, int8)


# 449 rows and more of 2560 channels are more 64-row tiles than SMs in every launch of a layer: the rows are cut again for the turns of the persistent
# kernel, differently for wide and narrow layers (att.output and ffn.value: 35 and 40 rows of int8, 65 and 74 of fp16)
@pytest.mark.parametrize("quant", [0, 1])
def test_step_of_rows_cut_for_turns_agrees_with_the_cpu_path(tmp_path, quant):
    p = rsv.write_synthetic(str(tmp_path / "m.st"), "tiny", seed=1, quant=quant, n_layer=1, n_embd=2560, n_head=40, ffn_hidden=5120, vocab=300, w_mid=24, a_mid=40,
                            v_mid=8, g_mid=72)
    b, o = rsv.ModelBuilder(p).build(), orc.OracleModel(p)
    for n in (449, 512):
        toks = np.random.default_rng(n).integers(0, 300, size=n).astype(np.uint32)
        b.reset()
        o.reset()
        lg, want = b.infer_seq(toks), o.forward(toks)
        # fp32 through the layer in another summation order: a few ulps of the logits' scale
        assert float(np.sqrt(np.mean((lg - want) ** 2))) <= 64 * 2.0 ** -24 * max(1.0, float(np.abs(want).max())), n
        assert np.abs(b.state_back() - o.state_back()).max() <= 1e-4 * max(1.0, float(np.abs(o.state_back()).max()))
    b.state.close()
    b.model.close()


# The smallest steps whose rows are cut again (10240 ffn channels): ffn.key of int8 weights has three tiles of 22 to 43 rows up to 128 rows; fp16 keeps its
# 64-row tiles there for one segment, has one tile where every row is a segment (93 rows and more), and three tiles from 129 rows on
@pytest.mark.parametrize("quant", [0, 1])
def test_small_steps_cut_for_turns_agree_with_the_cpu_path(tmp_path, quant):
    p = rsv.write_synthetic(str(tmp_path / "m.st"), "tiny", seed=2, quant=quant, n_layer=1, n_embd=2560, n_head=40, ffn_hidden=10240, vocab=300, w_mid=24, a_mid=40,
                            v_mid=8, g_mid=72)
    b, o = rsv.ModelBuilder(p).build(), orc.OracleModel(p)
    for n in (65, 80, 97, 128, 129, 193):
        toks = np.random.default_rng(n).integers(0, 300, size=n).astype(np.uint32)
        b.reset()
        o.reset()
        lg, want = b.infer_seq(toks), o.forward(toks)
        # fp32 through the layer in another summation order: a few ulps of the logits' scale
        assert float(np.sqrt(np.mean((lg - want) ** 2))) <= 64 * 2.0 ** -24 * max(1.0, float(np.abs(want).max())), n
        assert np.abs(b.state_back() - o.state_back()).max() <= 1e-4 * max(1.0, float(np.abs(o.state_back()).max()))
    for n in (65, 112, 128):
        toks = np.random.default_rng(n).integers(0, 300, size=n).astype(np.uint32)
        st = b.model.create_batch_state(n)
        got = b.model.forward_seq_batch_mean_hidden(st, [toks[i:i + 1] for i in range(n)])
        st.close()
        for i in range(0, n, 7):
            o.reset()
            want = o.mean_hidden(toks[i:i + 1])
            assert float(np.sqrt(np.mean((got[i] - want) ** 2))) <= 64 * 2.0 ** -24 * max(1.0, float(np.abs(want).max())), (n, i)
    b.state.close()
    b.model.close()


# 444 rows of 2560 channels are three LayerNorm blocks per SM of 148, 445 more than that (a block with fewer registers)
def test_steps_around_three_layernorm_blocks_per_sm(tmp_path):
    p = rsv.write_synthetic(str(tmp_path / "m.st"), "tiny", seed=3, quant=1, n_layer=1, n_embd=2560, n_head=40, ffn_hidden=1024, vocab=300, w_mid=24, a_mid=40, v_mid=16, g_mid=56)
    b, o = rsv.ModelBuilder(p).build(), orc.OracleModel(p)
    rng = np.random.default_rng(11)
    for n in (443, 444, 445):
        toks = rng.integers(0, b.info().num_vocab, size=n).astype(np.uint32)
        b.reset()
        o.reset()
        lg, want = b.infer_seq(toks), o.forward(toks)
        assert float(np.sqrt(np.mean((lg - want) ** 2))) <= 64 * 2.0 ** -24 * max(1.0, float(np.abs(want).max())), n  # (as above)
    b.state.close()
    b.model.close()


# Eight heads: steps on either side of the lines between the two WKV kernels (five and six pairs per SM, ten and twelve, fifteen and eighteen; 148 SMs) give the tokens and states of the
# same sessions in batches of 31, which stay below all of them
@pytest.mark.parametrize("sessions", [(92, 93), (111, 112), (184, 185), (222, 223), (277, 278), (333, 334)])
def test_sessions_around_the_wkv_lines(tiny_paths, sessions):
    m = rsv.ModelBuilder(tiny_paths["int8"]).build().model
    seeds = np.random.default_rng(5).integers(0, m.info().num_vocab, size=sessions[1]).astype(np.uint32)

    def stream(part):
        s = m.create_batch_state(len(part))
        toks = m.collect_sample_selfloop_batch(m.submit_sample_selfloop_batch(s, part, 6, None))
        return toks, [s.slot_back(i) for i in range(len(part))]

    parts = [stream(seeds[i:i + 31]) for i in range(0, len(seeds), 31)]
    few, states = np.concatenate([t for t, _ in parts]), [x for _, p in parts for x in p]
    for n in sessions:
        toks, got = stream(seeds[:n])
        assert np.array_equal(toks, few[:n])
        for i in range(n):
            assert float(np.sqrt(np.mean((got[i] - states[i]) ** 2))) <= 64 * 2.0 ** -24 * max(1.0, float(np.abs(states[i]).max())), (n, i)  # (as above)


# 184 sessions of 8 heads go to the WKV kernel of one block per pair, 186 to the one that streams pairs (the line is ten pairs per SM: 185)
def test_sessions_around_the_wkv_line(tiny_paths):
    m = rsv.ModelBuilder(tiny_paths["int8"]).build().model
    seeds = np.random.default_rng(5).integers(0, m.info().num_vocab, size=186).astype(np.uint32)

    def stream(part):
        s = m.create_batch_state(len(part))
        return m.collect_sample_selfloop_batch(m.submit_sample_selfloop_batch(s, part, 6, None))

    few = np.concatenate([stream(seeds[i:i + 31]) for i in range(0, 186, 31)])
    assert np.array_equal(stream(seeds), few) and np.array_equal(stream(seeds[:184]), few[:184])
