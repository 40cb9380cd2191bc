"""Logits on their way to the caller: pageable, pinned and device memory, chunks that go through the staging area and its threads, and
chunks that are too small for it."""
import ctypes
import os

import numpy as np
import pytest

import rwkv_rsv_b200 as rsv

pytestmark = pytest.mark.gpu

V = 16384  # a chunk of 64 positions and more is staged (2^20 logits)


@pytest.fixture(scope="module")
def bundle(model_dir):
    p = rsv.write_synthetic(os.path.join(model_dir, "vocab16k.st"), "tiny", seed=0, quant=0, n_layer=2, n_embd=256, n_head=4, ffn_hidden=1024, vocab=V, w_mid=16,
                            a_mid=16, v_mid=16, g_mid=16)
    return rsv.ModelBuilder(p).build()


def _full(b, toks, out_ptr):
    t = np.ascontiguousarray(toks, dtype=np.uint32)
    b.reset()
    if rsv.native().rsv_infer_full(b.model._h, b.state._h, t.ctypes.data_as(ctypes.c_void_p), t.size, ctypes.c_void_p(out_ptr)) != 0:
        raise rsv.RsvError(rsv.native().rsv_last_error().decode())


# 63 / 64: below and at the size that is staged; 140, 201: one staged chunk; 300: a staged chunk, then a small one
@pytest.mark.parametrize("n", [1, 63, 64, 140, 201, 300])
def test_logits_of_every_position(bundle, n):
    import torch
    b = bundle
    toks = np.random.default_rng(n).integers(0, V, size=n).astype(np.uint32)
    b.reset()
    want = np.stack([b.infer_chunked(toks[i:i + 1], 1) for i in range(n)])  # position by position, one row each
    pageable = np.full((n, V), np.nan, np.float32)
    _full(b, toks, pageable.ctypes.data)
    scale = max(1.0, float(np.abs(want).max()))
    # fp32 through two layers in another summation order
    assert np.abs(pageable - want).max() <= 64 * 2.0 ** -24 * scale
    pinned = torch.full((n, V), float("nan"), pin_memory=True)
    _full(b, toks, pinned.data_ptr())
    assert np.array_equal(pinned.numpy(), pageable)


# passes are 256 positions: up to the last one, one more, and three staged chunks in turn
@pytest.mark.parametrize("n", [255, 256, 257, 600])
def test_logits_of_every_position_around_a_pass(bundle, n):
    test_logits_of_every_position(bundle, n)


def test_logits_into_memory_of_the_device(bundle):
    # the arrays are the host's by contract; a device array is a matter for the driver's copy and never for the host's own
    import torch
    b = bundle
    toks = np.arange(70, dtype=np.uint32)
    host = np.empty((70, V), np.float32)
    _full(b, toks, host.ctypes.data)
    dev = torch.zeros((70, V), device="cuda")
    torch.cuda.synchronize()
    _full(b, toks, dev.data_ptr())
    assert np.array_equal(dev.cpu().numpy(), host)
    one = torch.zeros(V, device="cuda")
    torch.cuda.synchronize()
    t = np.array([3], dtype=np.uint32)
    b.reset()
    assert rsv.native().rsv_infer_tokens(b.model._h, b.state._h, t.ctypes.data_as(ctypes.c_void_p), 1, ctypes.c_void_p(one.data_ptr())) == 0
    b.reset()
    assert np.array_equal(one.cpu().numpy(), b.infer_tokens(t))
