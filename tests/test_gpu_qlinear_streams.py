"""What a single layer's handle keeps between calls: the status word of its bounded waits."""
import numpy as np
import pytest

from conftest import random_qlinear

pytestmark = pytest.mark.gpu


def make(l2, K, N, gs, seed=3):
    rng = np.random.default_rng(seed)
    return rng, l2.QLinear(*random_qlinear(rng, K, N, gs), gs)


@pytest.mark.parametrize("B", [2, 65, 600])  # the buffers of the first call, and larger ones
def test_recorded_failure_is_reported_once(l2, B):
    rng, q = make(l2, 256, 264, 64)
    x = rng.standard_normal((B, 256)).astype(np.float32)
    q.matvec(x[:2])
    want = q.matvec(x)
    _, q = make(l2, 256, 264, 64)
    q.matvec(x[:2])
    l2.check(l2.lib.l2_debug_qlinear_status(q._h, 2003))  # as an asynchronous call on device buffers would leave it
    with pytest.raises(l2.L2Error, match="2003"):
        q.matvec(x)
    assert np.array_equal(q.matvec(x), want)
    assert np.array_equal(q.matvec(x[0]), make(l2, 256, 264, 64)[1].matvec(x[0]))
