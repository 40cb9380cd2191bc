"""Checkpoints whose matrices do not all have one format: the format is the tensor's, so any mix of fp16, int8 with one (scale, zero) per
row and int8 with one per row and group loads and runs at every step size."""
import os

import numpy as np
import pytest

import orc
import rwkv_rsv_b200 as rsv
from checkpoint_files import read_safetensors, write_safetensors

pytestmark = pytest.mark.gpu

BIG = ("att.receptance", "att.key", "att.value", "att.output", "ffn.key", "ffn.value")
SHAPE = dict(n_layer=3, n_embd=512, n_head=8, ffn_hidden=2048, vocab=1000, w_mid=32, a_mid=32, v_mid=16, g_mid=64)


def _sources(tmp_path, **shape):
    return {name: read_safetensors(rsv.write_synthetic(os.path.join(str(tmp_path), name + ".st"), "tiny", seed=0, quant=q, **shape))
            for name, q in (("fp16", 0), ("int8", 1), ("int8g", 2))}


def _take(dst, src, prefix):
    """The matrix `prefix` (+ ".weight") of `dst` in the format it has in `src`."""
    for key in [k for k in dst if k.startswith(prefix + ".weight")]:
        del dst[key]
    for key in src:
        if key.startswith(prefix + ".weight"):
            dst[key] = src[key]


def _check(path, sizes, vocab):
    b, o = rsv.ModelBuilder(path).build(), orc.OracleModel(path)
    rng = np.random.default_rng(3)
    try:
        for n in sizes:
            toks = rng.integers(0, vocab, size=n).astype(np.uint32)
            b.reset()
            o.reset()
            lg, want = b.infer_seq(toks), o.forward(toks)
            # fp32 through the layers in another summation order: a few ulps of the logits' scale per layer
            assert float(np.sqrt(np.mean((lg - want) ** 2))) <= 64 * 2.0 ** -24 * max(1.0, float(np.abs(want).max())), n
            assert np.abs(b.state_back() - o.state_back()).max() <= 1e-4 * max(1.0, float(np.abs(o.state_back()).max()))
    finally:
        b.state.close()
        b.model.close()


# which format each of the three layers has
@pytest.mark.parametrize("layers", [("fp16", "int8", "int8"), ("int8", "fp16", "int8"), ("int8g", "int8", "fp16"), ("fp16", "int8g", "int8")])
def test_layers_of_different_formats(tmp_path, layers):
    src = _sources(tmp_path, **SHAPE)
    out = dict(src["fp16"])
    for i, fmt in enumerate(layers):
        for m in BIG:
            _take(out, src[fmt], f"blocks.{i}.{m}")
    _check(write_safetensors(os.path.join(str(tmp_path), "mixed.st"), out), (1, 2, 3, 16, 64, 65, 130), SHAPE["vocab"])


# a per-group file in which some matrices have the same (scale, zero) in every group of a row, so that they are rows with one: alone, and
# next to an fp16 matrix in the same launch
@pytest.mark.parametrize("uniform,half", [(("att.receptance",), ()), (("att.key", "att.value", "ffn.key"), ("att.receptance",)), ((), ("att.value",))])
def test_uniform_matrices_in_a_per_group_file(tmp_path, uniform, half):
    src = _sources(tmp_path, **SHAPE)
    out = dict(src["int8g"])
    for i in range(SHAPE["n_layer"]):
        for m in uniform:
            _take(out, src["int8"], f"blocks.{i}.{m}")
        for m in half:
            _take(out, src["fp16"], f"blocks.{i}.{m}")
    _check(write_safetensors(os.path.join(str(tmp_path), "uniform.st"), out), (2, 33, 64), SHAPE["vocab"])


def test_padding_of_the_last_k_block(tmp_path):
    """fp16 ffn.value whose K ends inside a block of 64, next to int8 matrices: what another step's operands left behind the K end must not
    reach the products."""
    shape = dict(SHAPE, n_layer=2)
    src = _sources(tmp_path, **shape)
    out = read_safetensors(rsv.write_synthetic(os.path.join(str(tmp_path), "f200.st"), "tiny", seed=0, quant=0, **dict(shape, ffn_hidden=200)))
    for i in range(2):
        for m in ("att.receptance", "att.key", "att.value", "att.output"):
            _take(out, src["int8"], f"blocks.{i}.{m}")
    _check(write_safetensors(os.path.join(str(tmp_path), "mixed.st"), out), (64, 2, 3, 5, 17, 130, 2, 33), shape["vocab"])


@pytest.mark.parametrize("quant", [1, 2])
def test_rows_wider_than_one_block(tmp_path, quant):
    """n_embd above 8192: a row no longer fits the LayerNorm kernel's block of 1024 threads with eight channels each."""
    shape = dict(n_layer=1, n_embd=8320, n_head=130, ffn_hidden=256, vocab=64, w_mid=16, a_mid=16, v_mid=16, g_mid=16)
    path = rsv.write_synthetic(os.path.join(str(tmp_path), "wide.st"), "tiny", seed=0, quant=quant, **shape)
    _check(path, (1, 3, 40), shape["vocab"])
    os.remove(path)


# ... and rows of 4160 and 8192 channels, which a block of 520 and of 1024 threads holds, also with more rows than are resident at once
@pytest.mark.parametrize("n_embd,sizes", [(4160, (1, 3, 40, 445)), (8192, (3, 40))])
def test_rows_of_one_large_block(tmp_path, n_embd, sizes):
    shape = dict(n_layer=1, n_embd=n_embd, n_head=n_embd // 64, ffn_hidden=256, vocab=64, w_mid=16, a_mid=16, v_mid=16, g_mid=16)
    path = rsv.write_synthetic(os.path.join(str(tmp_path), "block.st"), "tiny", seed=0, quant=0 if n_embd % 128 else 1, **shape)
    _check(path, sizes, shape["vocab"])
    os.remove(path)


# Per-group weights at the edges of their kernel: one group a row, odd numbers of them (also where K is split), 80; full and ragged row tiles of up to 32 rows; a vocabulary head whose
# last weight tile is partial and whose rows are no multiple of four
@pytest.mark.parametrize("n_embd,ffn,vocab", [(128, 128, 301), (384, 1408, 200), (640, 10240, 130)])
def test_groups_at_the_edges_of_a_tile(tmp_path, n_embd, ffn, vocab):
    shape = dict(n_layer=2, n_embd=n_embd, n_head=n_embd // 64, ffn_hidden=ffn, vocab=vocab, w_mid=16, a_mid=24, v_mid=16, g_mid=40)
    path = rsv.write_synthetic(os.path.join(str(tmp_path), "g.st"), "tiny", seed=0, quant=2, quant_head=True, **shape)
    _check(path, (1, 2, 3, 7, 8, 9, 29, 31, 32, 33, 65, 130), vocab)
