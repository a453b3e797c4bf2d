"""Calls one after the other with no wait between them, on one stream and on two in turn:
each reads what the call before wrote, or overwrites what it read. The chain kernels and
their preparations may begin while the kernel before still runs, so these orders rest on
their own waits. Every result equals that of the same calls with a wait after each."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

LINKS = 24


@pytest.fixture(scope="module", autouse=True)
def fg():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import flashgemm_b200 as fg
    fg.lib()
    fg.set_semantics("ref")
    fg.set_chain_mode("fused")
    fg.set_f32_algo("3xtf32")
    fg.set_narrow("always")
    yield fg
    fg.set_narrow("auto")


def _run(fg, links, buffers, streams, wait=False, copies=True):
    """The links in turn, each on the next of the streams; each link's result (copies) and
    the buffers' last state."""
    import torch
    for b, first in buffers:
        b.copy_(first)
    torch.cuda.synchronize()
    out = []
    for i, (call, result) in enumerate(links):
        with torch.cuda.stream(streams[i % len(streams)]):
            call()
            if wait:
                torch.cuda.synchronize()
            if copies:
                out.append(result.clone())
    torch.cuda.synchronize()
    fg.sync()
    return [t.cpu().numpy() for t in out], [b.cpu().numpy() for b, _ in buffers]


def _check(fg, links, buffers):
    import torch
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    want, end = _run(fg, links, buffers, [one], wait=True)
    assert all(np.isfinite(w).all() and w.any() for w in want + end)
    for _ in range(3):  # nothing at all between the calls
        got = _run(fg, links, buffers, [one], copies=False)[1]
        for x, y in zip(got, end):
            np.testing.assert_array_equal(x, y)
    got, last = _run(fg, links, buffers, [one, two])
    for x, y in zip(got + last, want + end):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("registered", [True, False], ids=["registered", "weights-split-per-call"])
@pytest.mark.parametrize("N", [4000, 30000])
def test_f32_chains_feed_each_other(fg, N, registered):
    """x -> y -> x -> ...: every call reads the C of the one before and overwrites its B."""
    import torch
    dims = [288, 96, 24, 288]
    g = torch.Generator(device="cuda").manual_seed(N)
    A = [torch.randn(m, k, generator=g, device="cuda") / k ** 0.5 for k, m in zip(dims, dims[1:])]
    W = [fg.Weights("f32", a) for a in A]
    x, y = torch.empty(288, N, device="cuda"), torch.empty(288, N, device="cuda")
    first = torch.randn(288, N, generator=g, device="cuda")

    def link(c, b):
        s = torch.cuda.current_stream
        if registered:
            return lambda: fg.chain_registered("f32", c, b, N, W, stream=s())
        return lambda: fg.chain_dev("f32", c, b, N, A, dims[1:], dims[:-1], stream=s())

    before = fg.kernel_launches()
    link(y, first)()
    assert fg.kernel_launches() - before == (1 if registered else 2)  # the column chain, the split
    links = [(link(y, x), y) if i % 2 == 0 else (link(x, y), x) for i in range(LINKS)]
    _check(fg, links, [(x, first), (y, torch.zeros_like(y))])
    for w in W:
        w.release()


def test_bf16_and_int8_chains_around_f32_ones(fg):
    """A BF16 chain writes what an FP32 chain reads, and the next one overwrites it; INT8
    chains whose weights are prepared per call run in between."""
    import torch
    N = 16384
    rng = np.random.default_rng(3)
    Bh, Ah, _ = oracle.chain_inputs("bf16", N, 256, [64, 40, 96], seed=11)
    bf = [fg.Weights("bf16", torch.from_numpy(a.view(np.int16)).cuda()) for a in Ah]
    bB = [torch.from_numpy(np.roll(Bh, i, axis=1).copy().view(np.int16)).cuda() for i in range(2)]
    g = torch.Generator(device="cuda").manual_seed(5)
    fd = [96, 48, 24, 64]
    fW = [fg.Weights("f32", torch.randn(m, k, generator=g, device="cuda") / k ** 0.5)
          for k, m in zip(fd, fd[1:])]
    Ms, Ks = [64, 40, 100], [128, 64, 40]
    iA = [torch.from_numpy(rng.integers(-127, 128, (m, k)).astype(np.int8)).cuda() for m, k in zip(Ms, Ks)]
    iB = torch.from_numpy(rng.integers(-127, 128, (128, N)).astype(np.int8)).cuda()
    mid = torch.empty(96, N, device="cuda")
    out = [torch.empty(64, N, device="cuda") for _ in range(LINKS // 3)]
    iC = torch.empty(100, N, dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream
    links = []
    for i in range(LINKS // 3):
        links += [(lambda i=i: fg.chain_registered("bf16", mid, bB[i % 2], N, bf, stream=s()), mid),
                  (lambda: fg.chain_dev("int8", iC, iB, N, iA, Ms, Ks, stream=s()), iC),
                  (lambda i=i: fg.chain_registered("f32", out[i], mid, N, fW, stream=s()), out[i])]
    _check(fg, links, [(mid, torch.zeros_like(mid)), (iC, torch.zeros_like(iC))] +
           [(o, torch.zeros_like(o)) for o in out])
    for w in bf + fW:
        w.release()
