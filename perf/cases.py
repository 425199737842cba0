"""What this framework is measured on: a set of calls that a user's program makes, from the smallest to the largest.

Six kinds of case, all through the package's public entry points:

  step      Megakernel.run(n): n training steps in one persistent launch (forward, backward, AdamW), fp32 char model or bf16 GPT
  decode    Megakernel.run(n) of a serving-only context: n greedy tokens, batch 1, KV cache
  eval      forward pass of a batch handed over by the host, logits read back
  layer     one transformer layer, forward and backward, as an explicit list of phases (run_phases)
  attention causal attention, forward and backward (run_phases)
  ln_bwd    LayerNorm backward with its dgamma on the caller's stream (ofa_ln_bwd_noalloc)

The bf16 path has one width (d_model 768, head dim 64), the fp32 path another (64, 16); vocabulary, depth, context length, batch,
number of rows and the options vary.
"""
import ctypes
import importlib
import threading

import numpy as np
import torch

ofa = importlib.import_module("open-flapping-airplanes_b200")
K = ofa.capi
DEV = "cuda"
D, FF, H = 768, 3072, 12          # bf16 path
SD, SH = 64, 4                    # fp32 path


def step(name, dtype, vocab, layers, ctx, batch, steps, tied=False, grad_bf16=False, serve=False):
    return {"name": name, "kind": "step", "dtype": dtype, "vocab": vocab, "layers": layers, "ctx": ctx, "batch": batch, "steps": steps,
            "tied": tied, "grad_bf16": grad_bf16, "serve": serve}


def decode(name, dtype, vocab, layers, ctx, sms, prompt, answer, tokens):
    return {"name": name, "kind": "decode", "dtype": dtype, "vocab": vocab, "layers": layers, "ctx": ctx, "sms": sms, "prompt": prompt,
            "answer": answer, "tokens": tokens}


def listed():
    return [
        # a host that already owns the GPU calls LayerNorm backward alone, on a ragged number of rows
        {"name": "ln_bwd_ragged", "kind": "ln_bwd", "rows": 1003, "dres": True, "accumulate": False},
        # the char-level model of the first configuration: one step at a time, the weights looked at after each
        step("char_step", "f32", 65, 2, 64, 16, 1),
        # and its 64-token greedy answer from an 8-token prompt
        decode("char_decode", "f32", 65, 2, 64, 0, 8, 64, 64),
        # a small bf16 model while a recipe is being debugged: few tokens, launches and phase changes are what it costs
        step("small_step", "bf16", 1152, 3, 384, 1, 2),
        # GPT-S, training only, all SMs: the flagship workload
        step("gpt_s_step", "bf16", 50304, 12, 1024, 4, 8),
        # the same beside a decode job that serves from the live weights (116 / 24 / 8 SMs)
        step("gpt_s_step_serving", "bf16", 50304, 12, 1024, 4, 8, serve=True),
        # tied head, large vocabulary, short context; gradients in the bf16 format of the all-reduce buckets
        step("tied_step", "bf16", 100352, 12, 512, 8, 4, tied=True, grad_bf16=True),
        # serving GPT-S from the whole GPU: one 6-token prompt and its 256-token answer
        decode("gpt_s_decode", "bf16", 50304, 12, 1024, 0, 6, 256, 261),
        # the same from the serving partition of the split
        decode("gpt_s_decode_24sm", "bf16", 50304, 12, 1024, 24, 6, 256, 261),
        # evaluation: the logits of a short batch of the host's tokens
        {"name": "gpt_s_eval", "kind": "eval", "vocab": 50304, "layers": 12, "ctx": 256, "batch": 1},
        # one layer at the GPT-S shape through an explicit phase list
        {"name": "layer_tasks", "kind": "layer", "ctx": 1024, "batch": 4},
        # attention alone over a long context
        {"name": "attention_long", "kind": "attention", "ctx": 4096, "batch": 1},
    ]


def _log(rng, lo, hi, multiple=1):
    v = lo * (hi / lo) ** rng.random()
    return max(lo, min(hi, round(v / multiple) * multiple))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "char", "decode", "decode", "eval", "layer", "attention", "ln_bwd"])
    if kind == "ln_bwd":
        return {"kind": "ln_bwd", "rows": _log(rng, 1, 32768), "dres": rng.random() < 0.7, "accumulate": rng.random() < 0.3}
    if kind == "attention":
        batch = rng.choice([1, 1, 2, 3, 4, 5, 8])
        return {"kind": "attention", "ctx": _log(rng, 128, min(4096, 16384 // batch), 128), "batch": batch}
    if kind == "layer":
        return {"kind": "layer", "ctx": _log(rng, 128, 1024, 128), "batch": rng.randint(1, 8)}
    if kind == "eval":
        batch = rng.randint(1, 2)
        return {"kind": "eval", "vocab": _log(rng, 512, 50304, 128), "layers": rng.randint(1, 12), "ctx": 128 * rng.randint(1, 4 // batch), "batch": batch}
    if kind == "char":
        c = step("", "f32", rng.randint(33, 300), rng.randint(1, 4), rng.randint(17, 96), rng.randint(1, 32), rng.choice([1, 1, 2, 5]))
    elif kind == "decode" and rng.random() < 0.3:
        c = decode("", "f32", rng.randint(33, 300), rng.randint(1, 4), rng.randint(33, 96), 0, rng.randint(1, 16), rng.randint(8, 64), rng.randint(8, 128))
    elif kind == "decode":
        prompt, answer = rng.randint(1, 32), rng.randint(16, 256)
        c = decode("", "bf16", _log(rng, 512, 50304, 128), rng.randint(1, 12), _log(rng, 384, 1024, 128), rng.choice([0, 0, 24, 16, 60]), prompt, answer,
                   prompt - 1 + answer)
    else:
        ctx = _log(rng, 128, 1024, 128)
        c = step("", "bf16", _log(rng, 512, 50304, 128), rng.randint(1, 12), ctx, rng.randint(1, min(8, 4096 // ctx)), rng.choice([1, 1, 2, 4, 8]),
                 tied=rng.random() < 0.4, grad_bf16=rng.random() < 0.4, serve=rng.random() < 0.3)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------ inputs
class _View:
    """Device memory of a context as a tensor, without a copy; the context lives as long as the tensor does."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (int(ptr), False), "version": 2}


def _grad_view(mk, bf16):
    v = torch.as_tensor(_View(mk, mk.grad_buffer_ptr(), (mk.num_params,), "<i2" if bf16 else "<f4"), device=DEV)
    return v.view(torch.bfloat16) if bf16 else v


def _config(case, mode):
    bf16 = case.get("dtype", "bf16") == "bf16"
    cfg = ofa.default_config("gpt_s" if bf16 else "tiny")
    cfg.vocab = cfg.valid_vocab = case["vocab"]
    cfg.n_layer, cfg.ctx_len, cfg.batch, cfg.mode = case["layers"], case["ctx"], case.get("batch", 1), mode
    cfg.decode_out_cap = 4096
    cfg.sched_profile = 0
    return cfg


def _create(cfg):
    """A context. The probe of the SMs that ofa_create runs on the new context's own stream can overtake the zero-fill of its buffers
    when other contexts are alive, and the call then fails: it is tried again, while a second thread allocates so that they meet otherwise."""
    try:
        return ofa.Megakernel(cfg)
    except ofa.OfaError:
        pass
    done = threading.Event()

    def allocate():
        while not done.is_set():
            ofa.DeviceBuffer((1 << 25,), "bf16").free()

    other = threading.Thread(target=allocate)
    other.start()
    try:
        for _ in range(100):
            try:
                return ofa.Megakernel(cfg)
            except ofa.OfaError:
                pass
    finally:
        done.set()
        other.join()
    return ofa.Megakernel(cfg)


def _load(mk, case, g, confident=False):
    """Weights of a freshly initialised model. `confident`: the head answers each token with one successor, as a trained model mostly
    does, so that a greedy answer does not hang on ties between near-equal logits."""
    w = torch.empty(mk.num_params, device=DEV).normal_(0.0, 0.02, generator=g)

    def span(name):
        off, n = mk.param_span(name)
        return w[off:off + n]

    span("gf").fill_(1.0)
    for layer in range(case["layers"]):
        for name in ("g1", "g2"):
            span(f"L{layer}.{name}").fill_(1.0)
        for name in ("Wo", "Wdn"):
            span(f"L{layer}.{name}").mul_((2 * case["layers"]) ** -0.5)
    if confident:
        width = mk.cfg.d_model
        wte, head = span("wte").view(-1, width), span("lm_head").view(-1, width)
        wte.mul_(50.0)
        successor = torch.randperm(wte.shape[0], generator=g, device=DEV)
        head[successor] += (0.02 if width == D else 0.1) * wte
    mk.load_weights(w.cpu().numpy())


def prepare(case, seed):
    kind = case["kind"]
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)

    def randn(*shape, scale=1.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, generator=g, device=DEV) * scale).to(dtype)

    if kind == "step":
        cfg = _config(case, K.MODE_TRAIN)
        cfg.tied_head, cfg.grad_bf16 = int(case["tied"]), int(case["grad_bf16"])
        cfg.data_seed = seed
        rng = np.random.default_rng(seed)
        if case["serve"]:
            cfg.infer_sms, cfg.reserved_sms, cfg.train_sms, cfg.use_decode = 24, 8, 116, 1
            cfg.n_prompt, cfg.answer_len, cfg.temperature = 6, 256, 0.0
            for i, t in enumerate(rng.integers(0, case["vocab"], 6)):
                cfg.prompt[i] = int(t)
        mk = _create(cfg)
        _load(mk, case, g)
        mk.set_tokens(rng.integers(0, case["vocab"], size=1 << 17, dtype=np.uint32))
        return {"case": case, "mk": mk, "grads": _grad_view(mk, case["grad_bf16"])}
    if kind == "decode":
        cfg = _config(case, K.MODE_DECODE_ONLY)
        cfg.use_decode, cfg.infer_sms, cfg.n_prompt, cfg.answer_len = 1, case["sms"], case["prompt"], case["answer"]
        for i, t in enumerate(np.random.default_rng(seed).integers(0, case["vocab"], case["prompt"])):
            cfg.prompt[i] = int(t)
        mk = _create(cfg)
        _load(mk, case, g, confident=True)
        return {"case": case, "mk": mk}
    if kind == "eval":
        mk = _create(_config(case, K.MODE_FORWARD))
        _load(mk, case, g)
        n = case["batch"] * (case["ctx"] + 1) + 1
        tokens = np.random.default_rng(seed).integers(0, case["vocab"], size=n, dtype=np.uint32)
        starts = (np.arange(case["batch"], dtype=np.uint32) * (case["ctx"] + 1))[None, :]
        return {"case": case, "mk": mk, "tokens": tokens, "starts": starts}
    if kind == "ln_bwd":
        n = case["rows"]
        x, dy = randn(n, D), randn(n, D)
        mean, var = x.float().mean(1), x.float().var(1, unbiased=False)
        dres = randn(n, D) if case["dres"] else None
        return {"case": case, "x": x, "dy": dy, "dres": dres, "gamma": (1.0 + randn(D, scale=0.1, dtype=torch.float32)).bfloat16(), "mean": mean.contiguous(),
                "rstd": torch.rsqrt(var + 1e-5).contiguous(), "dx": torch.empty_like(x), "dgamma": randn(D, dtype=torch.float32), "lib": K.load()}
    B, T = case["batch"], case["ctx"]
    N = B * T
    dims = dict(vocab=128, d_model=D, n_head=H, ctx_len=T, batch=B)
    t = {}

    def buf(name, *shape, dtype=torch.bfloat16):
        t[name] = torch.zeros(*shape, device=DEV, dtype=dtype)

    def ptr(*names):
        return [t[n].data_ptr() for n in names]

    for name, shape in (("qkv", (N, 3 * D)), ("att", (N, D)), ("datt", (N, D)), ("dqkv", (N, 3 * D))):
        buf(name, *shape)
    for name in ("lse", "Dr"):
        buf(name, B, H, T, dtype=torch.float32)
    if kind == "attention":
        t["qkv"], t["datt"] = randn(N, 3 * D), randn(N, D)
        phases = [ofa.phase(K.TK_ATT_FWD, ptr("qkv", "att", "lse")), ofa.phase(K.TK_ATT_PREP, ptr("att", "datt", "Dr")),
                  ofa.phase(K.TK_ATT_BWD, ptr("qkv", "datt", "lse", "Dr", "dqkv", "att"))]
        return {"case": case, "t": t, "dims": dims, "phases": phases, "out": ("att", "lse", "dqkv")}
    t["x"], t["dy"] = randn(N, D), randn(N, D, scale=1e-3)
    for name, shape in (("Wqkv", (D, 3 * D)), ("Wo", (D, D)), ("Wup", (D, FF)), ("Wdn", (FF, D))):
        t[name] = randn(*shape, scale=0.02)
        buf("d" + name, *shape, dtype=torch.float32)
    for name in ("g1", "g2"):
        t[name] = (1.0 + randn(D, scale=0.1, dtype=torch.float32)).bfloat16()
        buf("d" + name, D, dtype=torch.float32)
        buf("part_" + name, (N + 15) // 16, D, dtype=torch.float32)
        buf("mean_" + name, N, dtype=torch.float32)
        buf("rstd_" + name, N, dtype=torch.float32)
    for name in ("ln1", "h", "ln2", "y", "dln2", "dh", "dln1", "dx"):
        buf(name, N, D)
    for name in ("upre", "uact", "dpre"):
        buf(name, N, FF)

    def gemm(layout, epi, m, n, k, a, lda, b, ldb, c, ldc, aux=None, ldaux=0):
        return ofa.gemm_phase(layout, epi, m, n, k, t[a].data_ptr(), lda, t[b].data_ptr(), ldb, t[c].data_ptr(), ldc, t[aux].data_ptr() if aux else None, ldaux)

    NN, NT, TN = K.GEMM_NN, K.GEMM_NT, K.GEMM_TN
    row_term = gemm(NT, K.EPI_DR, N, D, D, "dh", D, "Wo", D, "datt", D, "att", D)
    row_term.p[4] = t["Dr"].data_ptr()
    phases = [
        ofa.phase(K.TK_LN_FWD, ptr("ln1", "mean_g1", "rstd_g1", "x", "g1")),
        gemm(NN, K.EPI_STORE, N, 3 * D, D, "ln1", D, "Wqkv", 3 * D, "qkv", 3 * D),
        ofa.phase(K.TK_ATT_FWD, ptr("qkv", "att", "lse")),
        gemm(NN, K.EPI_RES, N, D, D, "att", D, "Wo", D, "h", D, "x", D),
        ofa.phase(K.TK_LN_FWD, ptr("ln2", "mean_g2", "rstd_g2", "h", "g2")),
        gemm(NN, K.EPI_GELU, N, FF, D, "ln2", D, "Wup", FF, "uact", FF, "upre", FF),
        gemm(NN, K.EPI_RES, N, D, FF, "uact", FF, "Wdn", D, "y", D, "h", D),
        gemm(NT, K.EPI_DGELU, N, FF, D, "dy", D, "Wdn", D, "dpre", FF, "upre", FF),
        gemm(TN, K.EPI_F32, FF, D, N, "uact", FF, "dy", D, "dWdn", D),
        gemm(NT, K.EPI_STORE, N, D, FF, "dpre", FF, "Wup", FF, "dln2", D),
        gemm(TN, K.EPI_F32, D, FF, N, "ln2", D, "dpre", FF, "dWup", FF),
        ofa.phase(K.TK_LN_BWD, ptr("dh", "part_g2", "dln2", "h", "mean_g2", "rstd_g2", "g2", "dy")),
        ofa.phase(K.TK_LN_DG, ptr("dg2", "part_g2")),
        row_term,
        gemm(TN, K.EPI_F32, D, D, N, "att", D, "dh", D, "dWo", D),
        ofa.phase(K.TK_ATT_BWD, ptr("qkv", "datt", "lse", "Dr", "dqkv", "att")),
        gemm(NT, K.EPI_STORE, N, D, 3 * D, "dqkv", 3 * D, "Wqkv", 3 * D, "dln1", D),
        gemm(TN, K.EPI_F32, D, 3 * D, N, "ln1", D, "dqkv", 3 * D, "dWqkv", 3 * D),
        ofa.phase(K.TK_LN_BWD, ptr("dx", "part_g1", "dln1", "x", "mean_g1", "rstd_g1", "g1", "dh")),
        ofa.phase(K.TK_LN_DG, ptr("dg1", "part_g1")),
    ]
    return {"case": case, "t": t, "dims": dims, "phases": phases, "out": ("y", "dx", "dWqkv", "dWo", "dWup", "dWdn", "dg1", "dg2")}


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        mk = state["mk"]
        mk.run(case["steps"])
        out = {"losses": mk.losses()[-case["steps"]:], "grads": state["grads"]}
        if case["dtype"] == "f32":
            out["weights"] = mk.read_weights()   # the larger models' weights stay on the device, the next step's losses and gradients show them
        return out
    if kind == "decode":
        mk = state["mk"]
        mk.run(case["tokens"])
        return {"tokens": mk.decode_tokens(), "logits": mk.decode_logits()}
    if kind == "eval":
        mk = state["mk"]
        mk.set_tokens(state["tokens"])
        mk.set_starts(state["starts"])
        mk.run(1)
        return mk.read_buffer("logits", (case["batch"] * case["ctx"], case["vocab"]), "bf16")
    if kind == "ln_bwd":
        s = state
        rc = s["lib"].ofa_ln_bwd_noalloc(s["dx"].data_ptr(), s["dgamma"].data_ptr(), s["dy"].data_ptr(), s["x"].data_ptr(), s["mean"].data_ptr(), s["rstd"].data_ptr(),
                                         s["gamma"].data_ptr(), s["dres"].data_ptr() if s["dres"] is not None else None, case["rows"], D, int(case["accumulate"]),
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != K.OK:
            raise RuntimeError(s["lib"].ofa_noalloc_last_error().decode())
        return {"dx": s["dx"], "dgamma": s["dgamma"]}
    ofa.run_phases(K.DTYPE_BF16, state["dims"], state["phases"])
    return {k: state["t"][k] for k in state["out"]}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "ln_bwd":
        n = case["rows"] * D
        return {"bytes": (3 + case["dres"]) * 2 * n + 8 * case["rows"] + 2 * D + 4 * D * (1 + case["accumulate"]), "flops": 14 * n}
    if kind == "attention":
        n, pairs = case["batch"] * case["ctx"], case["batch"] * H * case["ctx"] ** 2 / 2
        return {"bytes": 2 * n * 8 * D + 4 * n * H, "flops": 3.5 * 4 * pairs * 64}
    if kind == "layer":
        n, pairs = case["batch"] * case["ctx"], case["batch"] * H * case["ctx"] ** 2 / 2
        return {"bytes": 2 * n * 4 * D + 12 * D * D * (2 + 4), "flops": 6 * n * 12 * D * D + 3.5 * 4 * pairs * 64}
    d, heads, size = (D, H, 2) if case.get("dtype", "bf16") == "bf16" else (SD, SH, 4)
    dh, L, V, T = d // heads, case["layers"], case["vocab"], case["ctx"]
    matmul = 12 * L * d * d + V * d
    if kind == "decode":
        mean_pos = min(case["prompt"] - 1 + case["answer"], T) / 2
        kv = 2 * L * d * size * mean_pos
        return {"bytes": case["tokens"] * (matmul * size + kv), "flops": case["tokens"] * (2 * matmul + 4 * L * d * mean_pos)}
    n = case["batch"] * T
    pairs = case["batch"] * heads * T * T / 2
    if kind == "eval":
        return {"bytes": 2 * matmul + 2 * n * V, "flops": 2 * n * matmul + 4 * L * pairs * dh}
    params = 12 * L * d * d + V * d * (1 if case.get("tied") else 2) + T * d
    per_param = 24 + (2 if case.get("grad_bf16") else 4) + (size if size == 2 else 0)   # master weight and two moments in and out, gradient out, working copy out
    return {"bytes": case["steps"] * params * per_param, "flops": case["steps"] * (6 * n * matmul + 3.5 * 4 * L * pairs * dh)}


def tolerance(case):
    if case.get("dtype") == "f32":
        return {"rel": 1e-4, "max": 0.05, "differ": 0.0}      # sums in another order, and AdamW's m / sqrt(v) of gradients near zero
    if case["kind"] == "decode":
        return {"rel": 1e-2, "max": 0.5, "differ": 0.0}       # logits of a bf16 model; the tokens are the same
    if case["kind"] == "ln_bwd":
        return {"rel": 4e-3, "max": 0.1}
    return {"rel": 2e-2, "max": 0.8}                          # bf16 activations and gradients through a deep model
