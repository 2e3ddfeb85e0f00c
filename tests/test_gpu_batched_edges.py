"""The batched QLinear (tcgen05) at the edges of its tiles: token blocks of 16 to 64, passes of 512, ragged rows and K steps,
slices of a cut tile, host arrays larger than the staging ring, device arrays off the 16-byte boundary; digits at their limits,
the ends of the f32 range, values that are not finite."""
import numpy as np
import pytest

from conftest import dequant_dense, random_qlinear

pytestmark = pytest.mark.gpu


def make(l2, K, N, gs, seed):
    rng = np.random.default_rng(seed)
    record = random_qlinear(rng, K, N, gs)
    return rng, l2.QLinear(*record, gs), dequant_dense(*record, gs)


def check(y, x, w, gs):
    # An activation is rounded by at most 2^-23 of its row's largest element (half a step); the group sums are exact; the rest is
    # f32: two roundings per group for the product and the sum, and a handful for scales, slices and factors.
    ax, aw = np.abs(x.astype(np.float64)), np.abs(w)
    groups = x.shape[1] // gs
    bound = 2.0**-23 * ax.max(axis=1, keepdims=True) * aw.sum(axis=1)[None] + (2 * groups + 8) * 2.0**-24 * (ax @ aw.T)
    err = np.abs(y.astype(np.float64) - x.astype(np.float64) @ w.T)
    assert (err <= bound).all(), "worst error over bound %.3g" % (err / bound).max()


# rows: one 8-row block, one row beyond a 256-row tile, several tiles; K: one group, a K step that is not full, several
@pytest.mark.parametrize("K,N,gs", [(32, 8, 32), (160, 264, 32), (192, 248, 64), (128, 256, 128), (1408, 520, 128), (4160, 4104, 64)])
def test_token_blocks(l2, K, N, gs):
    rng, q, w = make(l2, K, N, gs, K + N)
    for M in (2, 16, 17, 32, 33, 48, 49, 64, 65, 129):
        x = rng.standard_normal((M, K)).astype(np.float32) * np.exp(rng.uniform(-8, 8, (M, 1))).astype(np.float32)
        check(q.matvec(x), x, w, gs)


def test_several_passes_and_the_staging_ring(l2):
    import torch
    K, N, gs = 1024, 776, 64
    rng, q, w = make(l2, K, N, gs, 5)
    x = rng.standard_normal((1025, K)).astype(np.float32)  # 4 MB: four rounds of the ring; passes of 512, 512 and 1
    y = q.matvec(x)
    check(y, x, w, gs)
    # device arrays give the same bits, and so do pinned host arrays
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty(1025, N, device="cuda")
    q.matvec_dev(xd.data_ptr(), yd.data_ptr(), 1025, torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(yd.cpu().numpy(), y)
    assert np.array_equal(q.matvec(torch.from_numpy(x).pin_memory().numpy()), y)


@pytest.mark.parametrize("B", [1, 2, 37])
def test_device_arrays_off_the_16_byte_boundary(l2, B):
    import torch
    K, N, gs = 256, 264, 64
    rng, q, w = make(l2, K, N, gs, 9)
    x = rng.standard_normal((B, K)).astype(np.float32)
    st = torch.cuda.current_stream().cuda_stream
    want = torch.empty(B, N, device="cuda")
    xd = torch.from_numpy(x).cuda()
    q.matvec_dev(xd.data_ptr(), want.data_ptr(), B, st)
    check(want.cpu().numpy(), x, w, gs)
    for ox, oy in ((1, 0), (0, 1), (3, 2)):
        xs, ys = torch.zeros(B * K + 4, device="cuda"), torch.zeros(B * N + 4, device="cuda")
        xs[ox:ox + B * K] = xd.flatten()
        q.matvec_dev(xs.data_ptr() + 4 * ox, ys.data_ptr() + 4 * oy, B, st)
        assert torch.equal(ys[oy:oy + B * N].view(B, N), want)
        assert float(ys[:oy].abs().sum()) == 0 and float(ys[oy + B * N:].abs().sum()) == 0


# A group's sum at its limit: gs digits of one sign near (or at) 2048 against weights of magnitude 15 and 16.  The second group has
# weights 0: its activations only set the row's scale.  All factors are powers of two, so the result is that sum or it is wrong.
@pytest.mark.parametrize("gs", [32, 64, 128])
@pytest.mark.parametrize("digits", ["low", "high", "both"])
def test_group_sums_are_exact_at_their_limit(l2, gs, digits):
    K, N = 2 * gs, 264
    rng = np.random.default_rng(gs)
    q = np.zeros((N, K), np.uint32)  # q - z = -16 or -15 in the first group, 15 - 15 = 0 in the second
    if digits != "both":
        q[:, :gs] = rng.integers(0, 2, (N, gs))
    q[:, gs:] = 15
    qweight = np.zeros((N, K // 8), np.uint32)
    for j in range(8):
        qweight |= q[:, j::8] << np.uint32(4 * j)
    qzeros = np.zeros((N // 8, 2), np.uint32)
    qzeros[:, 0], qzeros[:, 1] = 0xFFFFFFFF, 0xEEEEEEEE  # z = nibble + 1
    perm = rng.permutation(K).astype(np.int32)
    layer = l2.QLinear(qweight.view(np.int32), qzeros.view(np.int32), np.full((N, 2), 0.5, np.float32), perm, gs)
    for M in (2, 33, 64):
        if digits == "both":
            X = np.full((M, K), 2**23 - 1, np.int64)  # digits 2048 and -1
        else:
            X = rng.integers(1900, 2048, (M, K)) * (4096 if digits == "high" else 1)
            X[:, gs:] = 5_000_000  # an exponent of 22, as the scale of both kinds of row
        X *= rng.choice([-1, 1], (M, 1))
        x = np.zeros((M, K), np.float32)
        shift = rng.integers(-40, 40, (M, 1))
        x[:, perm] = np.ldexp(X.astype(np.float64), shift)
        want = np.ldexp(X[:, :gs] @ (q[:, :gs].astype(np.int64) - 16).T * 0.5, shift)
        assert np.array_equal(layer.matvec(x).astype(np.float64), want)


def test_powers_of_two_change_nothing_but_the_exponent(l2):
    rng, q, w = make(l2, 256, 264, 64, 17)
    x = rng.standard_normal((33, 256)).astype(np.float32)
    y = q.matvec(x)
    for e in (-70, 64, 110, 120, 124):  # (at 124 the largest elements are about 2^126)
        assert np.array_equal(q.matvec(np.ldexp(x, e)), np.ldexp(y, e)), e


def test_rows_that_are_not_finite(l2):
    rng, q, w = make(l2, 256, 264, 64, 18)
    x = rng.standard_normal((33, 256)).astype(np.float32)
    y = q.matvec(x)
    x[3, 7], x[16, 255], x[32, 0] = np.nan, np.inf, -np.inf
    got = q.matvec(x)
    bad = np.isin(np.arange(33), (3, 16, 32))
    assert np.isnan(got[bad]).all()
    assert np.array_equal(got[~bad], y[~bad])
