"""What the host calls promise beside their results, on the GPU through the C ABI: a call has read its host buffers when it returns."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def pinned(n):
    t = torch.zeros(n, dtype=torch.int32, pin_memory=True)
    a = t.numpy().view(np.uint32)
    assert a.ctypes.data == t.data_ptr()
    return t, a


def tiny(ofa, mode, **fields):
    cfg = ofa.default_config("tiny")
    cfg.mode = mode
    for k, v in fields.items():
        setattr(cfg, k, v)
    mk = ofa.Megakernel(cfg)
    g = torch.Generator().manual_seed(7)
    mk.load_weights(torch.randn(mk.num_params, generator=g).mul_(0.05).numpy())
    return mk


def test_tokens_have_been_read_when_the_call_returns(ofa):
    """The source is page-locked and large, and its end, from which the windows are taken, is overwritten right after the call."""
    mk = tiny(ofa, ofa.capi.MODE_FORWARD)
    N, n = mk.cfg.batch * mk.cfg.ctx_len, 1 << 26
    starts = (n - 2048 + np.arange(mk.cfg.batch, dtype=np.uint32) * 70)[None, :]
    keep, tok = pinned(n)
    rng = np.random.default_rng(1)
    first, second = rng.integers(0, 65, 2048, dtype=np.uint32), rng.integers(0, 65, 2048, dtype=np.uint32)
    tok[-2048:] = first
    want = tok.copy()
    mk.set_tokens(want); mk.set_starts(starts); mk.run(1)
    ref = mk.read_buffer("logits", (N, 65), np.float32)
    mk.set_tokens(tok)
    tok[-2048:] = second
    mk.set_starts(starts); mk.run(1)
    np.testing.assert_array_equal(mk.read_buffer("logits", (N, 65), np.float32), ref)
    mk.close()


def test_starts_have_been_read_when_the_call_returns(ofa):
    mk = tiny(ofa, ofa.capi.MODE_FORWARD)
    B, N, rows = mk.cfg.batch, mk.cfg.batch * mk.cfg.ctx_len, 1 << 21
    rng = np.random.default_rng(2)
    mk.set_tokens(rng.integers(0, 65, 1 << 14, dtype=np.uint32))
    keep, st = pinned(rows * B)
    st = st.reshape(rows, B)
    st[-1] = np.arange(B) * 100
    zero = np.zeros(mk.num_params, np.float32)
    want = st.copy()
    mk.set_starts(want); mk.load_adam_state(zero, zero, rows - 1); mk.run(1)       # the step counter selects the table's last row
    ref = mk.read_buffer("logits", (N, 65), np.float32)
    mk.load_adam_state(zero, zero, rows - 1)
    mk.set_starts(st)
    st[-1] = 7 + np.arange(B) * 300
    mk.run(1)
    np.testing.assert_array_equal(mk.read_buffer("logits", (N, 65), np.float32), ref)
    mk.close()
