"""What the host calls promise beside their results, on the GPU through the C ABI: a call has read its host buffers when it returns, and
comes behind work that the caller queued on the default stream; reads work from several threads and where no thread can be started; launches
work again after a device reset, and what is kept between calls can be given back."""
import ctypes as C
import os
import subprocess
import sys
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


class _View:
    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (int(ptr), False), "version": 2}


def grads_of(mk, bf16):
    v = torch.as_tensor(_View(mk.grad_buffer_ptr(), mk.num_params, "<i2" if bf16 else "<f4"), device="cuda")
    return v.view(torch.bfloat16) if bf16 else v


def small_bf16(ofa, mode, grad_bf16=0):
    cfg = ofa.default_config("gpt_s")
    cfg.vocab = cfg.valid_vocab = 512
    cfg.n_layer, cfg.ctx_len, cfg.batch, cfg.mode, cfg.grad_bf16 = 1, 128, 1, mode, grad_bf16
    mk = ofa.Megakernel(cfg)
    g = torch.Generator().manual_seed(8)
    mk.load_weights(torch.randn(mk.num_params, generator=g).mul_(0.02).numpy())
    return mk


@pytest.mark.parametrize("bf16", [False, True])
def test_reads_are_ordered_behind_the_default_stream(ofa, bf16):
    """A host that scales the gradients through ofa_grad_buffer on the default stream reads the scaled ones."""
    mk = small_bf16(ofa, ofa.capi.MODE_NO_OPT, 1) if bf16 else tiny(ofa, ofa.capi.MODE_NO_OPT)
    mk.set_tokens(np.random.default_rng(3).integers(0, 65, 1 << 13, dtype=np.uint32))
    mk.run(1)
    before = mk.read_grads()
    g = grads_of(mk, bf16)
    torch.cuda._sleep(1000); g.mul_(1.0); torch.cuda.synchronize()       # both kernels are loaded: neither call below waits for the device
    torch.cuda._sleep(200_000_000)                   # about 0.1 s on the default stream
    g.mul_(2.0)
    np.testing.assert_array_equal(mk.read_grads(), 2.0 * before)
    mk.close()


def test_launches_are_ordered_behind_the_default_stream(ofa):
    """Gradients cleared on the default stream before a launch are cleared before it, not after its backward pass."""
    mk = tiny(ofa, ofa.capi.MODE_NO_OPT)
    mk.set_tokens(np.random.default_rng(4).integers(0, 65, 1 << 13, dtype=np.uint32))
    mk.set_starts(np.arange(mk.cfg.batch, dtype=np.uint32)[None, :] * 100)
    mk.run(1)
    before = mk.read_grads()
    g = grads_of(mk, False)
    torch.cuda._sleep(1000); g.zero_(); torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)
    g.zero_()
    mk.run(1)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(mk.read_grads(), before)
    mk.close()


def test_read_buffers_of_any_length_from_two_threads(ofa):
    """Lengths around the pieces a read is cut into (2 MB), odd counts among them, two contexts read at the same time."""
    SLOT = 2 << 20
    cases = []
    for seed in (1, 2):
        cfg = ofa.default_config("gpt_s")
        cfg.vocab = cfg.valid_vocab = 50304
        cfg.n_layer, cfg.ctx_len, cfg.batch, cfg.mode = 1, 128, 2, ofa.capi.MODE_FORWARD
        mk = ofa.Megakernel(cfg)
        g = torch.Generator().manual_seed(seed)
        w = torch.randn(mk.num_params, generator=g).mul_(0.02).numpy()
        mk.load_weights(w)
        mk.set_tokens(np.random.default_rng(seed).integers(0, 50304, 1 << 13, dtype=np.uint32))
        mk.run(1)
        cases.append((mk, w, mk.read_buffer("logits", (256 * 50304,), np.uint16)))
    errors = []

    def check(mk, w, bits):
        try:
            for n in (1, 3, SLOT // 2 - 1, SLOT // 2, SLOT // 2 + 1, 8 * SLOT // 2 + 5, 256 * 50304 - 1, 256 * 50304):
                wide = mk.read_buffer("logits", (n,), "bf16")
                np.testing.assert_array_equal(wide.view(np.uint32), bits[:n].astype(np.uint32) << 16)
                np.testing.assert_array_equal(mk.read_buffer("logits", (n,), np.uint16), bits[:n])
            for n in (1, SLOT // 4 + 1, mk.num_params - 3, mk.num_params):
                np.testing.assert_array_equal(mk._read(mk.lib.ofa_read_weights, n), w[:n])
        except BaseException as e:                   # shown by the test's own thread below
            errors.append(e)

    ts = [threading.Thread(target=check, args=c) for c in cases]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors[0]
    out = np.empty(4, np.float32)
    assert cases[0][0].lib.ofa_read_buffer_bf16(cases[0][0].h, b"logits", out.ctypes.data_as(C.c_void_p), (1 << 63) + 2) == ofa.capi.BAD_ARGUMENT
    for mk, _, _ in cases:
        mk.close()


SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
int refuse_threads = 0;
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
  static int (*real)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*) = 0;
  if (refuse_threads) return EAGAIN;
  if (!real) real = (int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*))dlsym(RTLD_NEXT, "pthread_create");
  return real(t, a, f, x);
}
"""


NO_THREADS = r"""
import ctypes, importlib, sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
ofa = importlib.import_module("open-flapping-airplanes_b200")
cfg = ofa.default_config("gpt_s")
cfg.vocab = cfg.valid_vocab = 8192
cfg.n_layer, cfg.ctx_len, cfg.batch, cfg.mode = 1, 128, 1, ofa.capi.MODE_FORWARD
mk = ofa.Megakernel(cfg)
w = torch.randn(mk.num_params, generator=torch.Generator().manual_seed(1)).mul_(0.02).numpy()
mk.load_weights(w)
flag = ctypes.c_int.in_dll(ctypes.CDLL(None), "refuse_threads")
flag.value = 1
got = mk.read_weights()
flag.value = 0
assert np.array_equal(got, w)
print("READ")
"""


def test_reads_work_where_no_thread_can_be_started(ofa, tmp_path):
    """pthread_create is replaced by one that fails, in a process of its own: no exception leaves the C entry, the weights arrive."""
    src, so, prog = tmp_path / "shim.c", tmp_path / "shim.so", tmp_path / "prog.py"
    src.write_text(SHIM); prog.write_text(NO_THREADS)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    r = subprocess.run([sys.executable, str(prog), ROOT], env=dict(os.environ, LD_PRELOAD=str(so)), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "READ" in r.stdout, (r.returncode, r.stdout[-500:], r.stderr[-2000:])


RESET = r"""
import ctypes, glob, importlib, os, sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
ofa = importlib.import_module("open-flapping-airplanes_b200")
K = ofa.capi
cands = glob.glob(os.path.join(os.path.dirname(os.path.dirname(torch.__file__)), "nvidia", "cuda_runtime", "lib", "libcudart.so*")) + ["libcudart.so.12", "/usr/local/cuda/lib64/libcudart.so"]
rt = None
for c in cands:
    try:
        rt = ctypes.CDLL(c); break
    except OSError:
        pass
w = np.random.default_rng(0).normal(0, 0.02, 1 << 20).astype(np.float32)
def once():
    for preset, V in (("tiny", 65), ("gpt_s", 512)):
        cfg = ofa.default_config(preset)
        cfg.vocab = cfg.valid_vocab = V
        if preset == "gpt_s": cfg.n_layer, cfg.ctx_len, cfg.batch = 1, 128, 1
        mk = ofa.Megakernel(cfg)
        mk.load_weights(np.resize(w, mk.num_params))
        mk.set_tokens(np.arange(4096, dtype=np.uint32) % V)
        mk.run(2)
        out = mk.losses(), mk.read_weights()
        mk.close()
        yield out
    dims = dict(vocab=65, d_model=64, n_layer=1, n_head=4, ctx_len=64, batch=4)
    a = ofa.DeviceBuffer.from_host(w[:4096].reshape(64, 64)); b = ofa.DeviceBuffer((64, 64), np.float32)
    ofa.run_phases(K.DTYPE_F32, dims, [ofa.gemm_phase(0, 0, 64, 64, 64, a, 64, a, 64, b, 64)])
    out = (b.download(),)
    a.free(); b.free()
    yield out
first = list(once())
rc = rt.cudaDeviceReset()
assert rc == 0, rc
second = list(once())
for x, y in zip(first, second):
    for p, q in zip(x, y):
        assert np.array_equal(p, q)
print("SAME")
"""


def test_everything_works_again_after_a_device_reset(ofa, tmp_path):
    prog = tmp_path / "prog.py"
    prog.write_text(RESET)
    r = subprocess.run([sys.executable, str(prog), ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "SAME" in r.stdout, (r.returncode, r.stdout[-500:], r.stderr[-2000:])


def test_what_calls_keep_is_bounded_and_can_be_given_back(ofa):
    """Ever larger phase lists push the smaller workspaces out; afterwards nothing of them is left."""
    lib, K = ofa.capi.load(), ofa.capi
    dims = dict(vocab=65, d_model=64, n_layer=1, n_head=4, ctx_len=64, batch=4)
    assert lib.ofa_release_caches() == K.OK
    free = torch.cuda.mem_get_info()[0]
    for n in (1, 40, 200, 500, 1000, 1500, 2000, 2500, 3, 3000):
        ofa.run_phases(K.DTYPE_F32, dims, [ofa.phase(K.TK_BARRIER)] * n)
        assert free - torch.cuda.mem_get_info()[0] <= 4 * (4 << 20) + (4 << 20)      # four of 4 MB, in granules of 2 MB
    assert lib.ofa_release_caches() == K.OK
    assert free - torch.cuda.mem_get_info()[0] <= 2 << 20
    assert ofa.run_phases(K.DTYPE_F32, dims, [ofa.phase(K.TK_BARRIER)] * 3) > 0
    assert lib.ofa_release_caches() == K.OK and lib.ofa_release_caches() == K.OK


def _gemm_case(ofa, K, N, Kd, seed):
    g = torch.Generator().manual_seed(seed)
    A, B = (torch.randn(256, Kd, generator=g) * 0.3).bfloat16(), (torch.randn(Kd, N, generator=g) * 0.3).bfloat16()
    bufs = [ofa.DeviceBuffer.from_host(A.float().numpy(), "bf16"), ofa.DeviceBuffer.from_host(B.float().numpy(), "bf16"), ofa.DeviceBuffer((256, N), "bf16")]
    return bufs, ofa.gemm_phase(0, 0, 256, N, Kd, bufs[0], Kd, bufs[1], N, bufs[2], N), (A.double() @ B.double()).numpy()


DIMS = dict(vocab=1024, d_model=768, n_layer=1, n_head=12, ctx_len=256, batch=2)


def test_a_workspace_is_reused_with_other_operands_shapes_sizes_and_threads(ofa):
    """Call after call through ofa_run_phases: other operands and shapes at the same place of the tables, phase lists and repeat counts
    that grow and shrink, from two threads. 256 x N x K products, bf16 results: half a unit in the last place of 8 bits, 2^-8 of the value."""
    K = ofa.capi
    errors = []

    def check(bufs, ref):
        got = bufs[2].download()
        assert np.abs(got - ref).max() <= 2.0 ** -8 * np.abs(ref).max() + 1e-3

    def work(base):
        try:
            torch.cuda.set_device(0)
            for i in range(24):
                cases = [_gemm_case(ofa, K, (128, 256, 384)[(i + j) % 3], (64, 192, 768)[(i + 2 * j) % 3], base + 100 * i + j) for j in range(1 + i % 5)]
                empty = [ofa.phase(K.TK_BARRIER)] * ((0, 3, 400, 7)[i % 4])
                ofa.run_phases(K.DTYPE_BF16, DIMS, [c[1] for c in cases] + empty, repeats=(1, 3, 600)[i % 3] if not empty else 1)
                for bufs, _, ref in cases:
                    check(bufs, ref)
        except BaseException as e:
            errors.append(e)

    ts = [threading.Thread(target=work, args=(b,)) for b in (1, 50000)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors[0]


def test_layernorm_backward_without_allocations_under_capture(ofa):
    """Both launches, the second a programmatic dependent one, recorded into a graph and replayed: the same bits as a direct call."""
    lib = ofa.capi.load()
    n, D = 1003, 768
    g = torch.Generator(device="cuda").manual_seed(5)
    x, dy = (torch.randn(n, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    gamma = torch.randn(D, generator=g, device="cuda").bfloat16()
    mean, rstd = x.float().mean(1), torch.rsqrt(x.float().var(1, unbiased=False) + 1e-5)

    def call(dx, dg):
        rc = lib.ofa_ln_bwd_noalloc(dx.data_ptr(), dg.data_ptr(), dy.data_ptr(), x.data_ptr(), mean.data_ptr(), rstd.data_ptr(), gamma.data_ptr(), None, n, D, 0,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == ofa.capi.OK, lib.ofa_noalloc_last_error().decode()

    want, wdg = torch.empty_like(x), torch.empty(D, device="cuda")
    call(want, wdg)
    torch.cuda.synchronize()
    dx, dg = torch.zeros_like(x), torch.zeros(D, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(dx, dg)
    for _ in range(3):
        dx.zero_(); dg.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(dx, want) and torch.equal(dg, wdg)
