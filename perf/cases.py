"""The work that a user has this framework do, as cases that can be timed and compared.

A case is one of

* ``step``      one token with the host in the loop (decode_step with logits), as an interactive program calls it;
* ``decode``    a run of tokens of the device-resident loop (decode_run) on a cache that holds a context;
* ``prompt``    a prompt up to its first own token: prefill, the positions the prefill ladder leaves to the
                one-token loop, and one decode_step that returns the logits (time to first token);
* ``generate``  generate_ids from a prompt to the last token, a fresh run state included;
* ``qlinear``   one quantised layer alone, QLinear.matvec on host arrays or matvec_dev on device tensors.

Model weights are the seeded synthetic checkpoint of the library (what every test and benchmark of the repository uses);
a program loads a model once and then serves many prompts, so a model stays loaded between the preparations of a process.
The seed decides the prompts, the activations and, for single layers, the weights.  The 7B shape runs at full depth.  The
13B and 70B shapes keep the first 10 of 40 and 8 of 80 layers: every layer does the same work, and the file stays quick.
"""
import os
import sys
from collections import OrderedDict

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "llama2.rs_b200"))
import llama2_rs as l2  # noqa: E402

WEIGHT_SEED = 20240
MODELS_KEPT = 6

# name: (preset or None, layers, group size)
NAMED = {"7B": (32, 128), "13B": (10, 128), "70B": (8, 64)}


def listed():
    return [
        # A small model answering a short prompt: latency of the calls, launches and set-up count, the weights fit the L2.
        dict(name="generate-small", kind="generate", model="generic", dim=1024, hidden=2816, layers=8, heads=8, kv_heads=2,
             vocab=8000, seq=512, gs=64, prompt=21, tokens=64),
        # Interactive use: one token at a time, the caller looks at the logits.
        dict(name="step-7b", kind="step", model="7B", context=160, temperature=0.0),
        # The headline configuration: 32-token prompt, 256 greedy tokens.
        dict(name="generate-7b", kind="generate", model="7B", prompt=32, tokens=256),
        # The end of a long conversation: the cache is nearly full, tokens are sampled.
        dict(name="decode-7b-context-1920", kind="decode", model="7B", context=1920, tokens=32, temperature=0.2),
        # Ordinary generation with the larger shapes (70B: grouped-query attention, group size 64).
        dict(name="decode-13b", kind="decode", model="13B", context=128, tokens=64, temperature=0.0),
        dict(name="decode-70b", kind="decode", model="70B", context=64, tokens=64, temperature=0.0),
        # A question's time to first token: short, ordinary with a ragged end, and a document.
        dict(name="prompt-7b-32", kind="prompt", model="7B", prompt=32),
        dict(name="prompt-13b-129", kind="prompt", model="13B", prompt=129),
        dict(name="prompt-70b-1536", kind="prompt", model="70B", prompt=1536),
        # One layer for callers that bring their own model: a vector, a ragged batch, a large batch.
        dict(name="qlinear-4096x11008-b1", kind="qlinear", k=4096, n=11008, gs=128, batch=1, host=False),
        dict(name="qlinear-5120x5120-b37-host", kind="qlinear", k=5120, n=5120, gs=128, batch=37, host=True),
        dict(name="qlinear-8192x28672-b256", kind="qlinear", k=8192, n=28672, gs=64, batch=256, host=False),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["step", "decode", "prompt", "prompt", "generate", "qlinear", "qlinear"])
    if kind == "qlinear":
        gs = rng.choice([32, 64, 128])
        while True:
            k, n = gs * max(1, _log(rng, 512, 28672) // gs), 8 * (_log(rng, 512, 28672) // 8)
            if k * n <= 8192 * 28672:
                break
        return dict(kind=kind, k=k, n=n, gs=gs, batch=_log(rng, 1, 256), host=rng.random() < 0.3)
    case = dict(kind=kind, model=rng.choice(["7B", "13B", "70B", "generic"]))
    seq = 2048
    if case["model"] == "generic":
        ag = rng.choice([1, 2, 4, 8])
        heads = ag * rng.randint(max(1, 4 // ag), max(1, 24 // ag))
        gs, seq = rng.choice([32, 64, 128]), rng.choice([512, 1024, 2048])
        case.update(dim=128 * heads, hidden=gs * int(128 * heads * rng.uniform(2.0, 3.5) // gs), layers=rng.randint(2, 8), heads=heads,
                    kv_heads=heads // ag, vocab=8 * rng.randint(250, 4000), seq=seq, gs=gs)
    if kind == "step":
        case.update(context=rng.randint(1, seq - 2), temperature=rng.choice([0.0, 0.2]))
    elif kind == "decode":
        tokens = _log(rng, 8, 128)
        case.update(context=rng.randint(1, seq - tokens), tokens=tokens, temperature=rng.choice([0.0, 0.0, 0.2]))
    elif kind == "prompt":
        case.update(prompt=_log(rng, 4, seq - 2))
    else:
        tokens = _log(rng, 8, 128)
        case.update(prompt=_log(rng, 2, seq - tokens - 2), tokens=tokens)
    return case


def _config(case):
    if case["model"] != "generic":
        layers, gs = NAMED[case["model"]]
        cfg = l2.preset_config(case["model"], gs)
        cfg.n_layers = layers
        return cfg
    cfg = l2.Config()
    cfg.dim, cfg.hidden_dim, cfg.n_layers, cfg.n_heads, cfg.n_kv_heads = case["dim"], case["hidden"], case["layers"], case["heads"], case["kv_heads"]
    cfg.vocab_size, cfg.seq_len, cfg.group_size = case["vocab"], case["seq"], case["gs"]
    return cfg


_models = OrderedDict()  # models that this process has loaded, the latest last


def _model(case):
    cfg = _config(case)
    key = repr(cfg)
    if key not in _models:
        while len(_models) >= MODELS_KEPT:
            _models.popitem(last=False)  # closed when the last state that uses it is gone
        _models[key] = l2.LlamaModel.synthetic(cfg, WEIGHT_SEED)
    _models.move_to_end(key)
    return _models[key]


def _random_qlinear(rng, k, n, gs):
    """A layer in the checkpoint's layout with the synthetic checkpoint's value distributions."""
    qweight = rng.integers(0, 2**32, size=(n, k // 8), dtype=np.uint32).view(np.int32)
    nibbles = rng.integers(6, 10, size=(n // 8, k // gs, 8), dtype=np.uint32)
    qzeros = np.zeros((n // 8, k // gs), np.uint32)
    for j in range(8):
        qzeros |= nibbles[:, :, j] << np.uint32(4 * j)
    scales = rng.random((n, k // gs), dtype=np.float32) * np.float32(0.018) + np.float32(0.002)
    return qweight, qzeros.view(np.int32), scales, rng.permutation(k).astype(np.int32)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "qlinear":
        k, n, b = case["k"], case["n"], case["batch"]
        layer = l2.QLinear(*_random_qlinear(rng, k, n, case["gs"]), case["gs"])
        x = rng.standard_normal((b, k), dtype=np.float32)
        if case["host"]:
            return dict(case=case, layer=layer, x=x)
        return dict(case=case, layer=layer, x=torch.from_numpy(x).cuda(), y=torch.zeros(b, n, device="cuda"))
    model = _model(case)
    vocab = model.config.vocab_size
    s = dict(case=case, model=model, seed=int(seed) + 1)
    if case["kind"] in ("step", "decode"):  # a conversation so far: `context` positions in the cache
        s["prompt"] = rng.integers(0, vocab, case["context"]).astype(np.int32)
        s["state"] = l2.RunState(model)
        first = l2.prefill(model, s["state"], s["prompt"])
        if first < case["context"]:
            l2.decode_run(model, s["state"], s["prompt"], first, case["context"])
    else:
        s["prompt"] = rng.integers(0, vocab, case["prompt"]).astype(np.int32)
        if case["kind"] == "prompt":
            s["state"] = l2.RunState(model)
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "qlinear":
        if case["host"]:
            return s["layer"].matvec(s["x"])
        s["layer"].matvec_dev(s["x"].data_ptr(), s["y"].data_ptr(), case["batch"], torch.cuda.current_stream().cuda_stream)
        return s["y"]
    model, prompt = s["model"], s["prompt"]
    if kind == "generate":
        r = l2.generate_ids(model, prompt, case["prompt"] + case["tokens"])
        return [r["tokens"], r["pos0"]]
    state = s["state"]
    if kind == "decode":
        random = l2.Random(s["seed"])
        tokens = l2.decode_run(model, state, prompt, case["context"], case["context"] + case["tokens"], case["temperature"], random)
        return tokens
    if kind == "step":
        token, logits = l2.decode_step(model, state, int(prompt[-1]), case["context"], case["temperature"], l2.Random(s["seed"]), want_logits=True)
        return [token, logits]
    first = l2.prefill(model, state, prompt)
    forced = l2.decode_run(model, state, prompt, first, case["prompt"])
    token, logits = l2.decode_step(model, state, int(prompt[-1]), case["prompt"], want_logits=True)
    return [forced, token, logits]


def _layer_weights(cfg):
    kv = cfg.dim // cfg.n_heads * cfg.n_kv_heads
    return 2 * cfg.dim * cfg.dim + 2 * cfg.dim * kv + 3 * cfg.dim * cfg.hidden_dim


def _quantised_bytes(weights, gs):
    return weights / 2 + weights / gs * 4.5  # nibbles; an f32 scale and a zero nibble per group


def _token_work(cfg, context):
    """One position of the one-token loop: all weights once, the classifier, the cache up to it."""
    kv = cfg.dim // cfg.n_heads * cfg.n_kv_heads
    w = _layer_weights(cfg) * cfg.n_layers
    cls = cfg.vocab_size * cfg.dim
    b = _quantised_bytes(w, cfg.group_size) + cls * 4 + cfg.n_layers * (context + 1) * kv * 2 * 4
    return b, 2 * (w + cls) + cfg.n_layers * (context + 1) * cfg.dim * 4


def _prefill_work(cfg, positions):
    """A prompt's batched positions: the layers' weights once, every cache row written once, causal attention."""
    kv = cfg.dim // cfg.n_heads * cfg.n_kv_heads
    w = _layer_weights(cfg) * cfg.n_layers
    if positions == 0:
        return 0, 0
    b = _quantised_bytes(w, cfg.group_size) + positions * cfg.dim * 4 + cfg.n_layers * positions * kv * 2 * 4
    return b, 2 * w * positions + cfg.n_layers * positions * (positions + 1) / 2 * cfg.dim * 4


def _ladder(n):
    """Positions of an n-token prompt that prefill takes; the one-token loop does the rest."""
    at = 0
    for step in (64, 32, 16, 8, 4, 2):
        while at + step < n:
            at += step
    return at


def work(case):
    kind = case["kind"]
    if kind == "qlinear":
        k, n, b = case["k"], case["n"], case["batch"]
        return {"bytes": _quantised_bytes(k * n, case["gs"]) + k * 4 + b * (k + n) * 4, "flops": 2 * k * n * b}
    cfg = _config(case)
    if kind in ("step", "decode"):
        positions, pre = range(case["context"], case["context"] + case.get("tokens", 1)), (0, 0)
    else:
        first = _ladder(case["prompt"])
        positions, pre = range(first, case["prompt"] + case.get("tokens", 1)), _prefill_work(cfg, first)
    parts = [pre] + [_token_work(cfg, p) for p in positions]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    # One layer is f32 sums of exact products.  Logits are f32 arithmetic through every layer of the model.  A chosen token is
    # a whole number; two equal logits, or a draw on the boundary of two tokens, may fall on either side.
    if case["kind"] == "qlinear":
        return {"rel": 1e-5}
    return {"rel": 5e-5, "differ": 0.01}
