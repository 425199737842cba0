"""Tasks at the sizes where their tiles, panels, rounds and task sizes end, on the GPU through the C ABI, against the CPU oracle."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

DIMS_T = dict(vocab=65, d_model=64, n_layer=1, n_head=4, ctx_len=64, batch=4)
EPS = 2.0 ** -24


def relmax(a, b):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-30)


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


@pytest.mark.parametrize("layout,M,N,Kd,pad", [
    (0, 33, 31, 65, 0), (0, 70, 65, 255, 1), (0, 64, 64, 256, 0), (0, 40, 100, 257, 3), (0, 32, 64, 515, 0),
    (1, 33, 31, 65, 0), (1, 64, 65, 255, 0), (1, 64, 64, 256, 0), (1, 31, 33, 300, 1), (1, 65, 64, 515, 2),
    (2, 17, 15, 127, 0), (2, 16, 16, 128, 0), (2, 65, 64, 129, 1), (2, 33, 48, 1, 0)])
def test_fp32_products_at_the_edges_of_their_panels(ofa, K, layout, M, N, Kd, pad):
    """k around one panel of 256 (NN, NT) and one round of 128 (TN), ragged tiles, rows of aligned and unaligned length. A result is a sum of
    k products: within (k + 2) * 2^-24 of the sum of their magnitudes, whatever the order."""
    g = torch.Generator().manual_seed(100 * layout + Kd)
    ash, bsh = ((M, Kd) if layout != 2 else (Kd, M)), ((Kd, N) if layout != 1 else (N, Kd))
    A, B = torch.randn(ash[0], ash[1] + pad, generator=g), torch.randn(bsh[0], bsh[1] + pad, generator=g)
    dA, dB, dC = ofa.DeviceBuffer.from_host(A.numpy()), ofa.DeviceBuffer.from_host(B.numpy()), ofa.DeviceBuffer((M, N + pad), np.float32)
    ofa.run_phases(K.DTYPE_F32, DIMS_T, [ofa.gemm_phase(layout, 0, M, N, Kd, dA, ash[1] + pad, dB, bsh[1] + pad, dC, N + pad)])
    a, b = A[:, :ash[1]].double(), B[:, :bsh[1]].double()
    a, b = (a if layout != 2 else a.T), (b if layout != 1 else b.T)
    got = dC.download()
    assert np.all(np.abs(got[:, :N] - (a @ b).numpy()) <= (Kd + 2) * EPS * (a.abs() @ b.abs()).numpy())
    assert not got[:, N:].any()


@pytest.mark.parametrize("T", [1, 17, 63, 64, 65, 96, 129, 150, 151])
def test_fp32_attention_around_its_rounds_of_64_rows(ofa, K, oracle, T):
    """151 is the longest context whose scores fit a block. Bounds as for the 64-row case."""
    B, H, dh = 2, 4, 16
    D, N = H * dh, 2 * T
    dims = dict(DIMS_T, ctx_len=T, batch=B)
    g = torch.Generator().manual_seed(T)
    qkv, dO = torch.randn(N, 3 * D, generator=g), torch.randn(N, D, generator=g)
    d_qkv, d_dO = ofa.DeviceBuffer.from_host(qkv.numpy()), ofa.DeviceBuffer.from_host(dO.numpy())
    d_o, d_lse, d_dqkv = ofa.DeviceBuffer((N, D), np.float32), ofa.DeviceBuffer((B, H, T), np.float32), ofa.DeviceBuffer((N, 3 * D), np.float32)
    ofa.run_phases(K.DTYPE_F32, dims, [ofa.phase(K.TK_ATT_FWD, [d_qkv, d_o, d_lse]), ofa.phase(K.TK_ATT_BWD, [d_qkv, d_dO, d_lse, None, d_dqkv, d_o])])
    o_ref, lse_ref = oracle.attention_ref(qkv, B, T, H, dh)
    assert relmax(d_o.download(), o_ref) <= 1e-5 and np.abs(d_lse.download() - lse_ref.numpy()).max() <= 1e-5
    assert relmax(d_dqkv.download(), oracle.attention_bwd_ref(qkv, dO, B, T, H, dh)) <= 1e-4


@pytest.mark.parametrize("V", [1, 31, 33, 2047, 2048, 2049, 5000])
def test_fp32_cross_entropy_on_both_sides_of_its_warp_form(ofa, K, V):
    dims = dict(DIMS_T, vocab=V, ctx_len=33, batch=1)
    N = 33
    g = torch.Generator().manual_seed(V)
    lg = torch.randn(N, V, generator=g) * 3; tg = torch.randint(0, V, (N,), generator=g, dtype=torch.int32)
    lg[:4] *= 5
    d_lg, d_tg, o_loss = ofa.DeviceBuffer.from_host(lg.numpy()), ofa.DeviceBuffer.from_host(tg.numpy()), ofa.DeviceBuffer((N,), np.float32)
    ofa.run_phases(K.DTYPE_F32, dims, [ofa.phase(K.TK_CE, [d_lg, d_tg, o_loss])])
    lgr = lg.clone().requires_grad_()
    l = F.cross_entropy(lgr, tg.long(), reduction="none"); l.mean().backward()
    assert np.abs(o_loss.download() - l.detach().numpy()).max() <= 1e-5 * max(1.0, float(l.abs().max()))
    assert np.abs(d_lg.download() - lgr.grad.numpy()).max() <= 1e-5 / N
