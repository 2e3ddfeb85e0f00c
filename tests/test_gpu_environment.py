"""What the environment holds does not make the library's results wrong."""
import numpy as np
import pytest

from conftest import random_qlinear, tiny_config

pytestmark = pytest.mark.gpu


# (builds of the token kernel for timing know them, see token_trace.py)
@pytest.mark.parametrize("name", ["L2_SK_SKIP", "L2_SK_NOCOPY"])
@pytest.mark.parametrize("flags", [0, 8])  # the token kernel; one launch per operator
def test_measuring_switches_are_not_in_the_library(l2, monkeypatch, name, flags):
    rng = np.random.default_rng(3)
    record, x = random_qlinear(rng, 256, 264, 64), rng.standard_normal(256).astype(np.float32)
    cfg = tiny_config(l2, n_layers=6)  # more weights than a CTA's ring holds, so that what is left in it is not the answer

    def results():
        model = l2.LlamaModel.synthetic(cfg, 5, flags=flags)
        return l2.QLinear(*record, 64).matvec(x), l2.transformer(model, l2.RunState(model), [9], [0])

    want = results()
    monkeypatch.setenv(name, "1")
    for got, ref in zip(results(), want):
        assert np.array_equal(got, ref)
