"""What a single layer's handle keeps between calls: the status word of its bounded waits, buffers that calls on several streams share,
the order with the default stream where no stream is given, first calls that wait for nobody, and inputs that the kernel in front has just written."""
import time

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


# (offset of the device arrays from the 16-byte boundary: batched calls on unaligned arrays go through the arrays of host calls)
@pytest.mark.parametrize("B,off", [(1, 0), (2, 0), (37, 0), (37, 1), (130, 3)])
@pytest.mark.parametrize("second", ["host", "stream"])
def test_calls_on_several_streams_take_turns(l2, B, off, second):
    import torch
    K, N = 1024, 776
    rng, q = make(l2, K, N, 64)
    xa, xb = rng.standard_normal((2, B, K)).astype(np.float32)
    want_a, want_b = q.matvec(xa), q.matvec(xb)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    da, db = torch.zeros(B * K + 4, device="cuda"), torch.zeros(B * K + 4, device="cuda")
    ya, yb = torch.zeros(B * N + 4, device="cuda"), torch.zeros(B * N + 4, device="cuda")
    da[off:off + B * K] = torch.from_numpy(xa).cuda().flatten()
    db[off:off + B * K] = torch.from_numpy(xb).cuda().flatten()
    torch.cuda.synchronize()
    for _ in range(3):
        with torch.cuda.stream(s1):
            torch.cuda._sleep(20_000_000)  # about 10 ms: the first call is still to come when the second is made
        q.matvec_dev(da.data_ptr() + 4 * off, ya.data_ptr() + 4 * off, B, s1.cuda_stream)
        if second == "host":
            got_b = q.matvec(xb)
        else:
            q.matvec_dev(db.data_ptr() + 4 * off, yb.data_ptr() + 4 * off, B, s2.cuda_stream)
        torch.cuda.synchronize()
        if second == "stream":
            got_b = yb[off:off + B * N].view(B, N).cpu().numpy()
        assert np.array_equal(got_b, want_b)
        assert np.array_equal(ya[off:off + B * N].view(B, N).cpu().numpy(), want_a)
        ya.zero_(), yb.zero_()
        torch.cuda.synchronize()


@pytest.mark.parametrize("B", [1, 37])
def test_captured_call(l2, B):
    import torch
    K, N = 1024, 776
    rng, q = make(l2, K, N, 64)
    x = rng.standard_normal((2, B, K)).astype(np.float32)
    want = [q.matvec(v) for v in x]  # (the first call allocates)
    xd, yd = torch.zeros(B, K, device="cuda"), torch.zeros(B, N, device="cuda")
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        q.matvec_dev(xd.data_ptr(), yd.data_ptr(), B, s.cuda_stream)
    for v, w in zip(x, want):
        xd.copy_(torch.from_numpy(v))
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(yd.cpu().numpy(), w)
        assert np.array_equal(q.matvec(v), w)


@pytest.mark.parametrize("B,off", [(1, 0), (37, 0), (37, 1)])
def test_no_stream_is_ordered_with_the_default_stream(l2, B, off):
    import torch
    K, N = 1024, 776
    rng, q = make(l2, K, N, 64)
    x = rng.standard_normal((B, K)).astype(np.float32)
    want = q.matvec(x)
    src = torch.from_numpy(x).cuda().flatten()
    xd, yd = torch.zeros(B * K + 4, device="cuda"), torch.zeros(B * N + 4, device="cuda")
    torch.cuda.synchronize()
    assert torch.cuda.current_stream().cuda_stream == 0
    for _ in range(3):
        torch.cuda._sleep(20_000_000)          # the input is not there yet when the call is made ...
        xd[off:off + B * K] = src
        q.matvec_dev(xd.data_ptr() + 4 * off, yd.data_ptr() + 4 * off, B)
        got = yd[off:off + B * N].clone()      # ... and the output is taken and both are overwritten without waiting on the host
        xd.zero_(), yd.zero_()
        assert np.array_equal(got.view(B, N).cpu().numpy(), want)


@pytest.mark.parametrize("B", [1, 2, 130])
def test_first_call_does_not_wait_for_other_work(l2, B):
    import torch
    K, N = 1024, 776
    rng, q = make(l2, K, N, 64)
    x = rng.standard_normal((B, K)).astype(np.float32)
    want = q.matvec(x)  # (the kernels are loaded)
    _, fresh = make(l2, K, N, 64)
    xd, yd = torch.from_numpy(x).cuda(), torch.zeros(B, N, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    busy = torch.cuda.Event()
    for st in (torch.cuda.default_stream(), s):
        with torch.cuda.stream(st):
            torch.cuda._sleep(600_000_000)  # about 0.3 s, on the default stream and on the call's
    busy.record(torch.cuda.default_stream())
    t = time.perf_counter()
    fresh.matvec_dev(xd.data_ptr(), yd.data_ptr(), B, s.cuda_stream)
    took = time.perf_counter() - t
    assert not busy.query() and took < 0.2
    torch.cuda.synchronize()
    assert np.array_equal(yd.cpu().numpy(), want)


@pytest.mark.parametrize("B", [1, 16, 64, 130])
def test_inputs_written_by_the_kernel_in_front(l2, B):
    # call after call on the same arrays, rows and their factors changing each time, nothing waited for in between
    import torch
    K, N = 1024, 776
    rng, q = make(l2, K, N, 64)
    x = rng.standard_normal((12, B, K)).astype(np.float32) * np.exp(rng.uniform(-6, 6, (12, B, 1))).astype(np.float32)
    want = np.stack([q.matvec(v) for v in x])
    s = torch.cuda.Stream()
    src, xd, yd = torch.from_numpy(x).cuda(), torch.zeros(B, K, device="cuda"), torch.zeros(B, N, device="cuda")
    got = torch.zeros(12, B, N, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        for i in range(12):
            torch.add(src[i], 0.0, out=xd)
            q.matvec_dev(xd.data_ptr(), yd.data_ptr(), B, s.cuda_stream)
            torch.add(yd, 0.0, out=got[i])
    torch.cuda.synchronize()
    assert np.array_equal(got.cpu().numpy(), want)
