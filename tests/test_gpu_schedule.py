"""Properties of the scheduler itself, on the GPU through the C ABI.

1. Order independence. The reference pulls the tasks of its libraries in shuffled orders and requires the same bits
   (llm/gemm/test_gemm.cu:20-49,238-278, llm/attention/test_attention.cu:45-77). Here the test hook
   ofa_debug_set_task_shuffle makes every phase hand out its tasks in a permuted order; GEMM, attention, LayerNorm,
   cross-entropy and embedding-backward outputs, and a whole training step, must not change by one bit.
2. Bounded waits. Every device-side wait gives up after a deadline and the kernel RETURNS with a status; nothing here
   faults or hangs a GPU: an external flag that nobody raises makes the wait run out (ST_EXTERNAL_TIMEOUT), ofa_abort
   stops a long launch, ofa_wait with a short timeout reports OFA_TIMEOUT and a later wait succeeds."""
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DIMS = dict(vocab=1024, d_model=768, n_layer=1, n_head=12, ctx_len=256, batch=2)


def bfr(t):
    return t.bfloat16().float()


def _task_chain(ofa):
    """one launch exercising every task kind whose result could depend on the order tasks are pulled in; returns output buffers"""
    K = ofa.capi
    V, D, T, B = DIMS["vocab"], DIMS["d_model"], DIMS["ctx_len"], DIMS["batch"]
    N = B * T
    g = torch.Generator().manual_seed(42)
    dev = lambda t, dt="bf16": ofa.DeviceBuffer.from_host(t.numpy(), dt)
    x = bfr(torch.randn(N, D, generator=g)); gamma = bfr(1 + 0.1 * torch.randn(D, generator=g))
    Wqkv = bfr(torch.randn(D, 3 * D, generator=g) * 0.05); Wh = bfr(torch.randn(V, D, generator=g) * 0.05)
    dO = bfr(torch.randn(N, D, generator=g)); tok = torch.randint(0, V, (N,), generator=g, dtype=torch.int32); tok[:40] = 3
    d_x, d_g, d_W, d_Wh, d_dO = dev(x), dev(gamma), dev(Wqkv), dev(Wh), dev(dO)
    d_tok = ofa.DeviceBuffer.from_host(tok.numpy(), np.int32)
    y = ofa.DeviceBuffer((N, D), "bf16"); mean = ofa.DeviceBuffer((N,), np.float32); rstd = ofa.DeviceBuffer((N,), np.float32)
    qkv = ofa.DeviceBuffer((N, 3 * D), "bf16"); o = ofa.DeviceBuffer((N, D), "bf16"); lse = ofa.DeviceBuffer((B, 12, T), np.float32)
    Dr = ofa.DeviceBuffer((B, 12, T), np.float32); dqkv = ofa.DeviceBuffer((N, 3 * D), "bf16")
    logits = ofa.DeviceBuffer((N, V), "bf16"); loss = ofa.DeviceBuffer((N,), np.float32)
    dW = ofa.DeviceBuffer((D, 3 * D), np.float32); dx = ofa.DeviceBuffer((N, D), "bf16"); part = ofa.DeviceBuffer(((N + 15) // 16, D), np.float32)
    dwte = ofa.DeviceBuffer((V, D), np.float32)
    phases = [
        ofa.phase(K.TK_LN_FWD, [y, mean, rstd, d_x, d_g]),
        ofa.gemm_phase(0, 0, N, 3 * D, D, y, D, d_W, 3 * D, qkv, 3 * D, nsub=2),
        ofa.phase(K.TK_ATT_FWD, [qkv, o, lse]),
        ofa.phase(K.TK_ATT_PREP, [o, d_dO, Dr]),
        ofa.phase(K.TK_ATT_BWD, [qkv, d_dO, lse, Dr, dqkv, o]),
        ofa.gemm_phase(2, 4, D, 3 * D, N, y, D, dqkv, 3 * D, dW, 3 * D),
        ofa.gemm_phase(1, 0, N, V, D, o, D, d_Wh, D, logits, V),
        ofa.phase(K.TK_CE, [logits, d_tok, loss]),
        ofa.phase(K.TK_LN_BWD, [dx, part, d_dO, d_x, mean, rstd, d_g, None]),
        ofa.phase(K.TK_EMB_WTE, [dwte, dx, d_tok], i0=0),
    ]
    ofa.run_phases(K.DTYPE_BF16, DIMS, phases)
    keep = [d_x, d_g, d_W, d_Wh, d_dO, d_tok]
    outs = {"y": y, "qkv": qkv, "o": o, "lse": lse, "dqkv": dqkv, "dW": dW, "dlogits": logits, "loss": loss, "dx": dx, "part": part, "dwte": dwte}
    return {k: (v.download().view(np.uint32) if v.dtype != "bf16" else v.download()).copy() for k, v in outs.items()}, keep


def test_task_order_does_not_change_any_bit(ofa):
    lib = ofa.capi.load()
    base, _ = _task_chain(ofa)
    assert np.isfinite(base["loss"].view(np.float32)).all()
    try:
        for seed in (1, 2024, 987654321):
            lib.ofa_debug_set_task_shuffle(seed)
            got, _ = _task_chain(ofa)
            for k in base:
                assert np.array_equal(got[k], base[k]), (seed, k)
    finally:
        lib.ofa_debug_set_task_shuffle(0)


def _small_training(ofa, oracle, nsteps=3):
    ocfg = oracle.OracleConfig(V=1024, D=768, L=2, H=12, T=256, B=2, tied=False)
    w0 = oracle.init_weights(ocfg)
    tokens = oracle.synthetic_tokens(ocfg.V, 1 << 15, 0)
    cfg = ofa.default_config("gpt_s")
    cfg.vocab, cfg.valid_vocab, cfg.n_layer, cfg.ctx_len, cfg.batch = ocfg.V, ocfg.V, ocfg.L, ocfg.T, ocfg.B
    return ocfg, w0, tokens, cfg


def test_training_steps_are_bitwise_identical_under_a_permuted_task_order(ofa, oracle):
    """also covers the hashed window starts (no starts table), which is what the benchmark uses"""
    lib = ofa.capi.load()
    ocfg, w0, tokens, cfg = _small_training(ofa, oracle)
    res = []
    try:
        for seed in (0, 31337):
            lib.ofa_debug_set_task_shuffle(seed)
            mk = ofa.Megakernel(cfg)
            mk.load_weights(oracle.flatten(ocfg, w0)); mk.set_tokens(tokens)
            mk.run(3, timeout_ms=120000)
            res.append((mk.losses().copy(), mk.read_weights().copy()))
            mk.close()
    finally:
        lib.ofa_debug_set_task_shuffle(0)
    assert np.array_equal(res[0][0].view(np.uint32), res[1][0].view(np.uint32))
    assert np.array_equal(res[0][1].view(np.uint32), res[1][1].view(np.uint32))
    # hashed starts: the first step's loss equals the oracle's on the windows the documented hash selects
    def splitmix64(z):
        m = (1 << 64) - 1
        z = (z + 0x9E3779B97F4A7C15) & m
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
        return z ^ (z >> 31)
    starts0 = np.array([[splitmix64(0 ^ (0 * ocfg.B + b)) % (len(tokens) - ocfg.T - 1) for b in range(ocfg.B)]], dtype=np.int64)
    ref = oracle.train(ocfg, w0, tokens, starts0, 1, precision="bf16_points")
    assert abs(res[0][0][0] - ref["losses"][0]) <= 1e-2 * ref["losses"][0]


def test_external_flag_that_nobody_raises_makes_the_wait_run_out(ofa, oracle):
    """ext_sync without a communication side: the graph raises "grads ready" and waits (bounded, 0.2 s here) for "allreduce done",
    which never comes. The kernel must RETURN with ST_EXTERNAL_TIMEOUT; the context can be destroyed and a fresh one trains."""
    ocfg, w0, tokens, cfg = _small_training(ofa, oracle)
    cfg.ext_sync, cfg.grad_bf16, cfg.timeout_s = 1, 1, 0.2
    mk = ofa.Megakernel(cfg)
    mk.load_weights(oracle.flatten(ocfg, w0)); mk.set_tokens(tokens)
    assert len(mk.buckets()) >= 2
    mk.launch(2)
    t0 = time.monotonic()
    with pytest.raises(ofa.OfaError) as e:
        mk.wait(20000)
    assert time.monotonic() - t0 < 10.0
    assert e.value.code == ofa.capi.DEVICE_ABORT and e.value.status.dev_code == 6        # ST_EXTERNAL_TIMEOUT
    name = mk.phases()[e.value.status.phase]["name"]
    assert name.startswith("allreduce done"), name
    assert mk.steps_done == 0
    mk.close()
    cfg.ext_sync, cfg.grad_bf16, cfg.timeout_s = 0, 0, 0.0
    ok = ofa.Megakernel(cfg)
    ok.load_weights(oracle.flatten(ocfg, w0)); ok.set_tokens(tokens)
    ok.run(2, timeout_ms=60000)
    assert np.all(np.isfinite(ok.losses())) and ok.steps_done == 2
    ok.close()


def test_abort_and_wait_timeout(ofa, oracle):
    ocfg, w0, tokens, cfg = _small_training(ofa, oracle)
    mk = ofa.Megakernel(cfg)
    mk.load_weights(oracle.flatten(ocfg, w0)); mk.set_tokens(tokens)
    mk.launch(20000)                                   # several seconds of work
    with pytest.raises(ofa.OfaError) as e:
        mk.wait(1)                                     # 1 ms: still running
    assert e.value.code == ofa.capi.TIMEOUT
    live = mk.live()
    assert mk.abort() == ofa.capi.OK
    t0 = time.monotonic()
    with pytest.raises(ofa.OfaError) as e:
        mk.wait(10000)
    assert time.monotonic() - t0 < 1.5, "the kernel did not return within a second of the abort request"
    assert e.value.code == ofa.capi.DEVICE_ABORT and e.value.status.dev_code == 0        # host-requested: no device-side failure recorded
    assert mk.abort() == ofa.capi.NOT_LAUNCHED
    # the context is still usable: an aborted launch does not count its steps, the next one runs to the end
    done_before = mk.steps_done
    mk.launch(300)
    with pytest.raises(ofa.OfaError) as e:
        mk.wait(0)
    assert e.value.code == ofa.capi.TIMEOUT
    mk.wait(60000)                                     # a later wait on the same launch succeeds
    assert mk.steps_done == done_before + 300
    assert live["steps"] >= 0
    mk.close()


@pytest.mark.parametrize("ctx,layers,vocab", [(1024, 12, 50304), (384, 3, 1152)])
def test_spread_adamw_gives_the_same_bits(ofa, ctx, layers, vocab):
    """A short batch spreads AdamW through the backward pass: losses and weights after two steps are those of the optimizer behind it."""
    out = []
    for spread in (0, -1):
        cfg = ofa.default_config("gpt_s")
        cfg.vocab = cfg.valid_vocab = vocab
        cfg.n_layer, cfg.ctx_len, cfg.batch, cfg.adam_interleave = layers, ctx, 1, spread
        mk = ofa.Megakernel(cfg)
        g = np.random.default_rng(3)
        mk.load_weights((g.standard_normal(mk.num_params, dtype=np.float32) * 0.02))
        mk.set_tokens(g.integers(0, vocab, size=1 << 14, dtype=np.uint32))
        mk.run(2)
        out.append((len(mk.phases()), mk.losses()[-2:].copy(), mk.read_weights()))
        mk.close()
    assert out[0][0] > out[1][0]
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("layers,vocab,ctx,batch,kw,env,shuffle", [
    (3, 8192, 384, 2, dict(tied_head=1, grad_bf16=1), None, 0),
    (3, 8192, 384, 2, dict(), None, 31337),
    (3, 1152, 384, 1, dict(), "OFA_B200_GLOBAL_RECS", 0),
    (16, 1152, 384, 1, dict(), None, 0),                                                            # 412 phases: more first tickets than fit the kernel parameter
    (3, 1152, 384, 1, dict(infer_sms=24, reserved_sms=8, train_sms=116, use_decode=1, n_prompt=6, adam_interleave=16), None, 0)])
def test_spread_adamw_gives_the_same_bits_in_every_form(ofa, monkeypatch, layers, vocab, ctx, batch, kw, env, shuffle):
    """Tied head with bf16 gradients, permuted task order, first tickets in global memory (asked for, or because they do not fit), live serving."""
    lib = ofa.capi.load()
    out = []
    if env:
        monkeypatch.setenv(env, "1")
    try:
        for spread in (kw.get("adam_interleave", 0), -1):
            lib.ofa_debug_set_task_shuffle(shuffle if spread >= 0 else 0)
            cfg = ofa.default_config("gpt_s")
            cfg.vocab = cfg.valid_vocab = vocab
            cfg.n_layer, cfg.ctx_len, cfg.batch = layers, ctx, batch
            for k, v in kw.items():
                setattr(cfg, k, v)
            cfg.adam_interleave = spread
            mk = ofa.Megakernel(cfg)
            g = np.random.default_rng(3)
            mk.load_weights(g.standard_normal(mk.num_params, dtype=np.float32) * 0.02)
            mk.set_tokens(g.integers(0, vocab, size=1 << 14, dtype=np.uint32))
            mk.run(3)
            out.append((len(mk.phases()), mk.losses()[-3:].copy(), mk.read_weights()))
            mk.close()
    finally:
        lib.ofa_debug_set_task_shuffle(0)
    assert out[0][0] > out[1][0]
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("preset", ["gpt_s", "tiny"])
@pytest.mark.parametrize("job", ["train", "serve", "both"])
def test_every_form_of_the_kernel_gives_the_same_bits(ofa, preset, job):
    """A launch that trains, serves or does both runs a kernel of its own, with or without time tables."""
    out = []
    for profile in (1, 0):
        cfg = ofa.default_config(preset)
        cfg.sched_profile = profile
        if preset == "gpt_s":
            cfg.vocab = cfg.valid_vocab = 1152
            cfg.n_layer, cfg.ctx_len, cfg.batch = 2, 256, 1
        if job != "train":
            cfg.use_decode, cfg.infer_sms, cfg.n_prompt, cfg.answer_len, cfg.temperature = 1, 24, 3, 16, 0.0
        if job == "serve":
            cfg.mode = ofa.capi.MODE_DECODE_ONLY
        elif job == "both":
            cfg.reserved_sms, cfg.train_sms = 8, 116
            cfg.lr_max = cfg.lr_min = 0.0              # the served weights do not move, so that what is served does not hang on timing
        mk = ofa.Megakernel(cfg)
        g = np.random.default_rng(5)
        mk.load_weights(g.standard_normal(mk.num_params, dtype=np.float32) * 0.02)
        res = {}
        if job != "serve":
            mk.set_tokens(g.integers(0, cfg.vocab, size=1 << 13, dtype=np.uint32))
        mk.run(40)
        if job != "serve":
            res["loss"], res["w"] = mk.losses()[-40:].copy(), mk.read_weights()
        if job != "train":
            t = np.asarray(mk.decode_tokens())
            res["tokens"] = t[t >= 0]                  # beside training, how many depends on how long the steps take
        out.append(res)
        mk.close()
    for k in out[0]:
        n = min(len(out[0][k]), len(out[1][k]))
        assert n > 0
        np.testing.assert_array_equal(out[0][k][:n], out[1][k][:n])


def _form(ofa, preset, job, profile=0, **kw):
    """A context of one kind of launch on the same partition of the SMs, weights and (training) tokens loaded; frozen weights unless told otherwise."""
    cfg = ofa.default_config(preset)
    cfg.sched_profile = profile
    if preset == "gpt_s":
        cfg.vocab = cfg.valid_vocab = 1152
        cfg.n_layer, cfg.ctx_len, cfg.batch = 2, 256, 1
    cfg.infer_sms, cfg.reserved_sms, cfg.train_sms, cfg.adam_interleave = 24, 8, 116, -1
    cfg.n_prompt, cfg.answer_len, cfg.temperature = 3, 16, 0.0
    cfg.lr_max = cfg.lr_min = 0.0
    cfg.use_decode = int(job != "train")
    if job == "serve":
        cfg.mode = ofa.capi.MODE_DECODE_ONLY
    for k, v in kw.items():
        setattr(cfg, k, v)
    mk = ofa.Megakernel(cfg)
    g = np.random.default_rng(5)
    mk.load_weights(g.standard_normal(mk.num_params, dtype=np.float32) * 0.02)
    if job != "serve":
        mk.set_tokens(g.integers(0, cfg.vocab, size=1 << 13, dtype=np.uint32))
    return mk


@pytest.mark.parametrize("tables", ["parameter", "global"])
@pytest.mark.parametrize("preset", ["gpt_s", "tiny"])
def test_kinds_of_launch_agree(ofa, monkeypatch, preset, tables):
    """What a launch that does both trains is what one that only trains does, what it serves is what one that only serves does; first tickets
    of both jobs in the kernel parameter or in global memory. No time tables."""
    if tables == "global":
        monkeypatch.setenv("OFA_B200_GLOBAL_RECS", "1")
    out = {}
    for job in ("train", "serve", "both"):
        mk = _form(ofa, preset, job)
        mk.run(40, timeout_ms=60000)
        if job != "serve":
            out[job, "loss"], out[job, "w"] = mk.losses()[-40:].copy(), mk.read_weights()
        if job != "train":
            t = np.asarray(mk.decode_tokens())
            out[job, "tokens"] = t[t >= 0]
        mk.close()
    np.testing.assert_array_equal(out["both", "loss"], out["train", "loss"])
    np.testing.assert_array_equal(out["both", "w"], out["train", "w"])
    n = min(len(out["both", "tokens"]), len(out["serve", "tokens"]))
    assert n > 0
    np.testing.assert_array_equal(out["both", "tokens"][:n], out["serve", "tokens"][:n])


@pytest.mark.parametrize("profile", [0, 1])
@pytest.mark.parametrize("preset,job", [("gpt_s", "serve"), ("gpt_s", "both"), ("tiny", "serve"), ("tiny", "both")])
def test_abort_of_a_launch_that_serves(ofa, preset, job, profile):
    """The abort word reaches a claim as a copy and a wait directly; the context can be used again."""
    mk = _form(ofa, preset, job, profile)
    n = 400000 if job == "serve" else 100000 if preset == "tiny" else 40000             # 8 s and more
    mk.launch(n)
    with pytest.raises(ofa.OfaError) as e:
        mk.wait(100)
    assert e.value.code == ofa.capi.TIMEOUT
    assert mk.abort() == ofa.capi.OK
    t0 = time.monotonic()
    with pytest.raises(ofa.OfaError) as e:
        mk.wait(10000)
    assert time.monotonic() - t0 < 1.5
    assert e.value.code == ofa.capi.DEVICE_ABORT and e.value.status.dev_code == 0
    mk.run(20, timeout_ms=60000)
    mk.close()


def test_expired_wait_of_a_launch_that_serves(ofa):
    """Serving alone, every wait given 1.5 us: one runs out, the kernel returns and says which (ST_DEP_TIMEOUT)."""
    mk = _form(ofa, "gpt_s", "serve", infer_sms=0, timeout_s=1e-6)
    mk.launch(2000)
    with pytest.raises(ofa.OfaError) as e:
        mk.wait(20000)
    assert e.value.code == ofa.capi.DEVICE_ABORT and e.value.status.dev_code == 1
    assert 0 <= e.value.status.phase < len(mk.decode_phases())
    mk.close()


def test_expired_external_wait_beside_a_serving_job(ofa):
    """The training job gives up (a flag that nobody raises); the serving blocks leave with it."""
    mk = _form(ofa, "gpt_s", "both", ext_sync=1, grad_bf16=1, timeout_s=0.2, adam_interleave=0)
    mk.launch(2)
    t0 = time.monotonic()
    with pytest.raises(ofa.OfaError) as e:
        mk.wait(20000)
    assert time.monotonic() - t0 < 5.0
    assert e.value.code == ofa.capi.DEVICE_ABORT and e.value.status.dev_code == 6 and mk.decode_steps > 0
    mk.close()


@pytest.mark.parametrize("ctx,profile", [(1152, 0), (2048, 0), (2048, 1)])
def test_waits_for_more_than_eight_row_blocks(ofa, oracle, monkeypatch, ctx, profile):
    """Beyond 1,024 tokens a sequence has more row blocks than a wait's lanes take at once: gradients against the oracle (bounds of the model
    tests), and the same bits in a permuted task order and when every dependency is of whole phases."""
    lib = ofa.capi.load()
    ocfg = oracle.OracleConfig(V=512, D=768, L=1, H=12, T=ctx, B=1, tied=False)
    w0 = oracle.init_weights(ocfg)
    tokens = oracle.synthetic_tokens(ocfg.V, 1 << 14, 0)
    starts = oracle.batch_starts(ocfg, 1 << 14, 1)
    cfg = ofa.default_config("gpt_s")
    cfg.vocab, cfg.valid_vocab, cfg.n_layer, cfg.ctx_len, cfg.batch, cfg.mode, cfg.sched_profile = ocfg.V, ocfg.V, 1, ctx, 1, ofa.capi.MODE_NO_OPT, profile
    got = []
    try:
        for seed, phase_deps in ((0, False), (4711, False), (0, True)):
            lib.ofa_debug_set_task_shuffle(seed)
            if phase_deps:
                monkeypatch.setenv("OFA_B200_PHASE_DEPS", "1")
            mk = ofa.Megakernel(cfg)
            mk.load_weights(oracle.flatten(ocfg, w0)); mk.set_tokens(tokens); mk.set_starts(starts.astype(np.uint32))
            mk.run(1, timeout_ms=60000)
            got.append((float(mk.losses()[0]), mk.read_grads()))
            spans = {n: mk.param_span(n) for n in ("wte", "wpe", "lm_head", "gf", "L0.g1", "L0.Wqkv", "L0.Wo", "L0.g2", "L0.Wup", "L0.Wdn")}
            mk.close()
    finally:
        lib.ofa_debug_set_task_shuffle(0)
    for loss, grads in got[1:]:
        assert loss == got[0][0]
        np.testing.assert_array_equal(grads, got[0][1])
    if profile:
        return
    ref = oracle.train(ocfg, w0, tokens, starts, 1, precision="bf16_points", grab_step0=True)
    assert abs(got[0][0] - ref["losses"][0]) <= 1e-2 * ref["losses"][0]
    gref = oracle.flatten(ocfg, ref["grads0"])
    for name, (off, cnt) in spans.items():
        a, b = got[0][1][off:off + cnt].astype(np.float64), gref[off:off + cnt].astype(np.float64)
        assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(b), name
