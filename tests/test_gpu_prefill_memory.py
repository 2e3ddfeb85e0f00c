"""A long prompt where the buffers of its largest batches do not fit the device beside what else is there: smaller batches."""
import numpy as np
import pytest

from conftest import assert_close, tiny_config

pytestmark = pytest.mark.gpu


def test_long_prompt_on_a_full_device(l2):
    import torch
    # batches of 512 need about 300 MB of this shape, of 256 half of that, of 64 about 40 MB
    cfg = tiny_config(l2, group_size=64, n_kv_heads=2, n_layers=1, dim=1024, hidden=28672, seq_len=1024)
    prompt = np.random.default_rng(8).integers(0, cfg.vocab_size, 611).astype(np.int32)

    def first_token(hold):
        model = l2.LlamaModel.synthetic(cfg, 6)
        state = l2.RunState(model)
        l2.decode_step(model, state, 1, 0, want_logits=True)  # what a token needs is there
        room = None
        if hold:
            torch.cuda.empty_cache()
            room = torch.empty(torch.cuda.mem_get_info()[0] - hold, dtype=torch.uint8, device="cuda")
            assert torch.cuda.mem_get_info()[0] <= hold
        at = l2.prefill(model, state, prompt)
        logits = []
        for p in range(at, len(prompt) + 1):
            logits.append(l2.decode_step(model, state, int(prompt[p - 1]), p, want_logits=True)[1])
        del room
        torch.cuda.empty_cache()
        return at, np.stack(logits)

    at, want = first_token(0)
    for hold in (130 << 20, 70 << 20):
        got_at, got = first_token(hold)
        assert got_at == at
        assert_close(got, want, rel=1e-4, abs_=1e-4, what="logits with %d MB free" % (hold >> 20))
