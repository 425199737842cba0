"""Tasks at the sizes where their tiles, panels, rounds and task sizes end, on the GPU through the C ABI, against the CPU oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K(ofa):
    return ofa.capi


@pytest.mark.parametrize("bf,V", [(True, 128), (True, 2432), (True, 4864), (True, 9600), (False, 1), (False, 7), (False, 65), (False, 1183), (False, 2400)])
def test_embedding_gradient_with_each_task_size(ofa, K, bf, V):
    """A task covers 8 to 128 rows of the vocabulary, by its size; ids at the edges of the tasks, repeated and absent ones."""
    D, T, B = (768, 128, 2) if bf else (64, 64, 4)
    N = T * B
    dims = dict(vocab=V, d_model=D, n_layer=1, n_head=12 if bf else 4, ctx_len=T, batch=B)
    g = torch.Generator().manual_seed(V)
    tok = torch.randint(0, V, (N,), generator=g, dtype=torch.int32)
    edge = [v for c in (8, 16, 32, 64, 128) for v in (c - 1, c, c + 1, 2 * c) if v < V] + [0, V - 1]
    tok[:len(edge)] = torch.tensor(edge, dtype=torch.int32); tok[N - len(edge):] = tok[:len(edge)]
    dx = torch.randn(N, D, generator=g)
    dx = dx.bfloat16().float() if bf else dx
    d_dx, d_tok, out = ofa.DeviceBuffer.from_host(dx.numpy(), "bf16" if bf else np.float32), ofa.DeviceBuffer.from_host(tok.numpy()), ofa.DeviceBuffer.from_host(np.full((V, D), 9.0, np.float32))
    ofa.run_phases(K.DTYPE_BF16 if bf else K.DTYPE_F32, dims, [ofa.phase(K.TK_EMB_WTE, [out, d_dx, d_tok])])
    ref = np.zeros((V, D), np.float32)
    for n in range(N):                                   # the order of the task: increasing position
        ref[tok[n]] += dx[n].numpy()
    np.testing.assert_array_equal(out.download(), ref)


@pytest.mark.parametrize("nsub", [0, 1, 4001, 4002, 4003])
def test_training_step_with_tasks_ordered_along_n(ofa, nsub):
    """A task waits for the producers of its rows and asks for its weights ahead, whatever the order of a phase's tasks: the gradients do not change."""
    cfg = ofa.default_config("gpt_s")
    cfg.vocab = cfg.valid_vocab = 640
    cfg.n_layer, cfg.ctx_len, cfg.batch, cfg.mode, cfg.gemm_nsub = 1, 256, 1, ofa.capi.MODE_NO_OPT, nsub
    mk = ofa.Megakernel(cfg)
    w = torch.randn(mk.num_params, generator=torch.Generator().manual_seed(3)).mul_(0.02).numpy()
    mk.load_weights(w); mk.set_tokens(np.random.default_rng(1).integers(0, 640, 1 << 13, dtype=np.uint32)); mk.set_starts(np.array([[17]], np.uint32))
    mk.run(1)
    got = mk.read_grads()
    mk.close()
    cfg.gemm_nsub = 2
    mk = ofa.Megakernel(cfg)
    mk.load_weights(w); mk.set_tokens(np.random.default_rng(1).integers(0, 640, 1 << 13, dtype=np.uint32)); mk.set_starts(np.array([[17]], np.uint32))
    mk.run(1)
    np.testing.assert_array_equal(got, mk.read_grads())
    mk.close()


@pytest.mark.parametrize("bf,gbf", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("off_out,off_in", [(0, 0), (1, 0), (0, 1), (2, 2), (3, 1)])
def test_position_gradient_at_any_element(ofa, K, bf, gbf, off_out, off_in):
    """Result and operand begin at any element of a buffer, as the scalar form of the task allowed."""
    D, T, B = (768, 128, 3) if bf else (64, 18, 5)
    dims = dict(vocab=128, d_model=D, n_layer=1, n_head=12 if bf else 4, ctx_len=T, batch=B)
    g = torch.Generator().manual_seed(1)
    dx = torch.randn(B * T, D, generator=g)
    dx = dx.bfloat16().float() if bf else dx
    src = ofa.DeviceBuffer.from_host(np.concatenate([np.zeros(off_in, np.float32), dx.numpy().ravel(), np.zeros(4, np.float32)]), "bf16" if bf else np.float32)
    out = ofa.DeviceBuffer.from_host(np.full(off_out + T * D + 4, 5.0, np.float32), "bf16" if gbf else np.float32)
    ofa.run_phases(K.DTYPE_BF16 if bf else K.DTYPE_F32, dims, [ofa.phase(K.TK_EMB_WPE, [out.at(off_out), src.at(off_in)], i1=1 if gbf else 0)])
    ref = np.zeros((T, D), np.float32)
    for b in range(B):
        ref += dx.numpy().reshape(B, T, D)[b]
    got = out.download()
    if gbf:
        ref = torch.from_numpy(ref).bfloat16().float().numpy()
    np.testing.assert_array_equal(got[off_out:off_out + T * D].reshape(T, D), ref)
    assert np.all(got[:off_out] == 5.0) and np.all(got[off_out + T * D:] == 5.0)
