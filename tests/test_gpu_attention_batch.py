"""The attention kernels of the batched forward, each by itself, against attention in 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HS = 128
HEAD, TILED, WIDE = 0, 1, 2


def attend(l2, kind, n_kv, q, kc, vc, pos):
    import torch
    M, n_heads = q.shape[:2]
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (q, kc, vc, pos.astype(np.int32))]
    out = torch.full((M, n_heads, HS), 7.0, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    l2.check(l2.lib.l2_debug_attention_batch(n_heads, n_kv, M, kind, *(t.data_ptr() for t in dev), out.data_ptr(), s.cuda_stream))
    torch.cuda.synchronize()
    return out.cpu().numpy()


def exact(n_kv, q, kc, vc, pos):
    """Result and a bound of the f32 error, [M][n_heads][HS]."""
    M, n_heads = q.shape[:2]
    q, kc, vc = (a.astype(np.float64) for a in (q, kc, vc))
    want, bound = np.zeros((M, n_heads, HS)), np.zeros((M, n_heads, HS))
    u = 2.0**-24
    for m in range(M):
        T = pos[m] + 1
        for h in range(n_heads):
            k, v = kc[:T, h * n_kv // n_heads], vc[:T, h * n_kv // n_heads]
            s = k @ q[m, h] / np.sqrt(HS)
            p = np.exp(s - s.max())
            p /= p.sum()
            want[m, h] = p @ v
            # a score is a sum of 128 products (128 roundings at most) and a quotient; its error, and that of the largest score, turns
            # up as a relative error of a probability, with a few roundings for expf; the sums over the positions and the rescalings
            # of the online softmax (one per tile) come on top
            score = 130 * u * (np.abs(k) @ np.abs(q[m, h])).max() / np.sqrt(HS)
            bound[m, h] = 2 * (2 * score + (T + T // 16 + 16) * u) * (p @ np.abs(v))
    return want, bound


# one token; tokens that do not fill a warp, a CTA, or exactly do; contexts that end inside, at the end and at the start of a tile of 32
@pytest.mark.parametrize("ag", [1, 2, 4, 8])
@pytest.mark.parametrize("kind", [HEAD, TILED, WIDE])
def test_against_64_bits(l2, ag, kind):
    rng = np.random.default_rng(10 * ag + kind)
    n_kv = 2
    per_cta = 64 // ag
    for M, last in ((1, 0), (1, 31), (1, 200), (2, 32), (per_cta - 1, 95), (per_cta, 96), (per_cta + 1, 223), (2 * per_cta + 3, 191)):
        if last + 1 < M:
            continue
        q = rng.standard_normal((M, n_kv * ag, HS)).astype(np.float32)
        kc, vc = rng.standard_normal((2, last + 1, n_kv, HS)).astype(np.float32)
        for pos in (np.arange(last + 1 - M, last + 1), rng.permutation(last + 1)[:M]):  # a prompt's positions; any others
            got = attend(l2, kind, n_kv, q, kc[:pos.max() + 1], vc[:pos.max() + 1], pos)
            want, bound = exact(n_kv, q, kc, vc, pos)
            err = np.abs(got - want)
            assert (err <= bound).all(), "M %d last %d: worst error over bound %.3g" % (M, last, (err / bound).max())


# a cache row that a query does not attend to may hold anything
@pytest.mark.parametrize("ag", [1, 2, 4, 8])
@pytest.mark.parametrize("kind", [HEAD, WIDE])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_rows_not_attended_to_do_not_matter(l2, ag, kind, value):
    rng = np.random.default_rng(ag)
    n_kv, M, T = 2, 64 // ag + 5, 150
    q = rng.standard_normal((M, n_kv * ag, HS)).astype(np.float32)
    kc, vc = rng.standard_normal((2, T, n_kv, HS)).astype(np.float32)
    pos = np.arange(T - M, T)
    want = attend(l2, kind, n_kv, q, kc, vc, pos)
    for row in (T - M // 2, T - 1):
        k2, v2 = kc.copy(), vc.copy()
        k2[row], v2[row] = value, value
        got = attend(l2, kind, n_kv, q, k2, v2, pos)
        assert np.array_equal(got[pos < row], want[pos < row])
        assert np.isnan(got[pos >= row]).all()
