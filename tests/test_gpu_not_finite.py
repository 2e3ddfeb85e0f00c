"""Values that are not finite do not turn into finite results: one row alone (B = 1), and a vector in the middle of the one-token forward."""
import numpy as np
import pytest

from conftest import random_qlinear, tiny_config

pytestmark = pytest.mark.gpu


# 32: one group; 12416: blocks beyond those a thread keeps in registers between the two passes over the vector
@pytest.mark.parametrize("K,gs", [(32, 32), (256, 64), (1408, 128), (12416, 128)])
def test_one_row(l2, K, gs):
    import torch
    rng = np.random.default_rng(K)
    layer = l2.QLinear(*random_qlinear(rng, K, 264, gs), gs)
    x = rng.standard_normal(K).astype(np.float32)
    y = layer.matvec(x)
    assert np.isfinite(y).all()
    for at in (0, K // 2, K - 1):
        for value in (np.nan, np.inf, -np.inf):
            bad = x.copy()
            bad[at] = value
            assert np.isnan(layer.matvec(bad)).all(), (at, value)
            xd, yd = torch.from_numpy(bad).cuda(), torch.zeros(264, device="cuda")
            layer.matvec_dev(xd.data_ptr(), yd.data_ptr(), 1, torch.cuda.current_stream().cuda_stream)
            assert bool(yd.isnan().all()), (at, value)
    assert np.array_equal(layer.matvec(x), y)  # and the next call is not touched by it
    x[0] = np.finfo(np.float32).max  # finite, and so is its product with a weight (below 16 * 0.02)
    assert np.isfinite(layer.matvec(x)).all()


def words(cfg):
    """Offsets (in 32-bit words of the payload) of the embedding and of the first scale of wv, wo, w1, w2, w3 in layer 0."""
    D, H, L, KV, gs = cfg.dim, cfg.hidden_dim, cfg.n_layers, cfg.dim // cfg.n_heads * cfg.n_kv_heads, cfg.group_size
    at, found = 1, {"embedding": 1}  # (the payload begins with the rmsnorm epsilon)
    at += cfg.vocab_size * D + L * D
    for name, n, k in (("wq", D, D), ("wk", KV, D), ("wv", KV, D), ("wo", D, D), ("norm", 0, 0), ("w1", H, D), ("w2", D, H), ("w3", H, D)):
        if name == "norm":
            at += L * D
            continue
        found[name] = at + n * k // 8 + n // 8 * (k // gs)
        at += L * (n * k // 8 + n // 8 * (k // gs) + n * (k // gs) + k)
    return found


# The vector that the value gets into first: wo's input through wv (no norm), w2's through w3 (no norm), those of wq, wk, wv and of w1, w3
# through the embedding and through wo (normed).
@pytest.mark.parametrize("gs", [32, 64, 128])
@pytest.mark.parametrize("where", ["wv", "w3", "embedding", "wo"])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("flags", [0, 8])  # the token kernel; one launch per operator
def test_in_the_forward(l2, orc, gs, where, value, flags):
    cfg = tiny_config(l2, group_size=gs, n_kv_heads=2)
    payload = l2.synth_fill(cfg, 41)
    token = 7
    at = words(cfg)[where] + (token * cfg.dim + 5 if where == "embedding" else 0)
    view = payload.view(np.float32)
    assert 0 < abs(view[at]) < 1  # a scale, or a value of the embedding
    view[at] = value
    gpu = l2.LlamaModel.from_blob(cfg, payload, flags=flags)
    cpu = orc.Model(cfg, payload)
    gs_, cs = l2.RunState(gpu), orc.State(cpu)
    logits, want = l2.transformer(gpu, gs_, [token], [0]), cpu.transformer(cs, [token], [0])
    assert not np.isfinite(want).any() and np.isnan(logits).all()
    for layer in range(cfg.n_layers):  # and what the cache keeps of it
        for got, ref in zip(gs_.read_kv(layer), cs.kv(layer)):
            assert np.array_equal(np.isfinite(got[0]), np.isfinite(ref[0])), layer
    assert 0 <= l2.decode_step(gpu, gs_, token, 1)[0] < cfg.vocab_size
