"""The plain FP32 SGEMM's tile shapes at the sizes where a tile can go wrong: edges
in M, N and K, K blocks of 2048 with remainders, rows and pointers that are not
16-byte aligned, on device memory. Bit for bit the oracle's result (one FMA per k
in increasing k, K cut into blocks of 2048), NaN and infinity included."""
import subprocess
import sys

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

# the launcher's shape for a 148-SM device beside each size
SIZES = [
    (31999, 1000, 17), (4096, 4096, 48),  # 64 x 128
    (1300, 1100, 65),   # 64 x 64
    (64, 18496, 31),    # 64 x 64, whole tiles
    (257, 4001, 33),    # 40 x 64
    (40, 6400, 32),     # 40 x 64, whole tiles
    (96, 4096, 100),    # 32 x 64
    (1, 1, 1), (17, 63, 2), (16, 64, 4), (129, 127, 15),  # 16 x 64
    (35, 457, 2049), (130, 260, 4100), (16, 16, 6144),    # K in blocks of 2048, side by side
    (1300, 1100, 2080),                                   # and in turn
]


def _device(a, offset):
    """The array on the device, its first element `offset` floats past an aligned address."""
    import torch
    buf = torch.zeros(a.size + offset + 4, device="cuda")
    t = buf[offset:offset + a.size].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("offsets", [(0, 0, 0), (1, 0, 0), (0, 2, 3)], ids=["aligned", "a", "bc"])
@pytest.mark.parametrize("shape", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
def test_sgemm_tiles_bitexact(shape, offsets):
    import torch
    import flashgemm_b200 as fg
    M, N, K = shape
    A, B = oracle.sgemm_inputs(M, N, K, seed=M + 3 * N + K)
    A[M // 2, K - 1] = np.inf   # the last k of a row: a k past it must not meet it
    B[K - 1, N // 2] = np.nan
    rows = sorted({0, 1 % M, M // 2, (M - 1) // 3, M - 1}) if M * N > 1 << 20 else list(range(M))
    want = oracle.sgemm_f32(np.ascontiguousarray(A[rows]), B, kblock=2048)
    a, b = _device(A, offsets[0]), _device(B, offsets[1])
    c = _device(np.full((M, N), 7.0, np.float32), offsets[2])
    fg.sgemm_dev(c, a, b, M, N, K)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(c.cpu().numpy()[rows], want)


@pytest.mark.parametrize("N", [(1 << 29) + 100, (1 << 29) + 101, 1 << 30],
                         ids=["2^29+100", "2^29+101", "2^30"])
def test_more_columns_than_a_31_bit_byte_count(N):
    """Rows of 2 GB and more, with and without 16-byte-aligned rows: every column is
    computed. Small whole numbers, so that every sum is exact."""
    import torch
    import flashgemm_b200 as fg
    M, K = 2, 2
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.tensor([[3.0, -2.0], [5.0, 7.0]], device="cuda")
    b = torch.randint(-8, 9, (K, N), generator=g, device="cuda", dtype=torch.int8).float()
    c = torch.full((M, N), 0.5, device="cuda")
    fg.sgemm_dev(c, a, b, M, N, K)
    torch.cuda.synchronize()
    for i in range(M):
        assert torch.equal(c[i], a[i, 0] * b[0] + a[i, 1] * b[1])


def test_captured_call_with_k_blocks():
    """K > 2048 on a stream that is being captured: no workspace, the blocks in turn, and
    the graph computes from what its operands hold when it runs."""
    import torch
    import flashgemm_b200 as fg
    M, N, K = 35, 457, 4100
    A, B = oracle.sgemm_inputs(M, N, K, seed=1)
    a, b = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    c = torch.zeros(M, N, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    fg.sgemm_dev(c, a, b, M, N, K, stream=s)  # the work is on this stream from here on
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        fg.sgemm_dev(c, a, b, M, N, K, stream=s)
    for scale in (1.0, -2.0):
        a.copy_(torch.from_numpy(A) * scale)
        c.fill_(7.0)
        graph.replay()
        torch.cuda.synchronize()
        want = oracle.sgemm_f32(A * np.float32(scale), B, kblock=2048)
        np.testing.assert_array_equal(c.cpu().numpy(), want)


NO_ROOM = """
import torch
import flashgemm_b200 as fg
M = N = 512
K = 800 * 2048                       # 838 MB of K-block sums
g = torch.Generator(device="cuda").manual_seed(5)
a = torch.rand(M, K, generator=g, device="cuda") - 0.5
b = torch.rand(K, N, generator=g, device="cuda") - 0.5
c = torch.zeros(M, N, device="cuda")
fg.sgemm_dev(c, a, b, M, N, 32)      # the kernels are loaded, and what every call needs is there
torch.cuda.synchronize()
torch.cuda.empty_cache()
filler = torch.empty(torch.cuda.mem_get_info()[0] - (400 << 20), dtype=torch.uint8, device="cuda")
fg.sgemm_dev(c, a, b, M, N, K)
torch.cuda.synchronize()
in_turn = c.clone()
del filler
torch.cuda.empty_cache()
c.zero_()
fg.sgemm_dev(c, a, b, M, N, K)
torch.cuda.synchronize()
assert torch.equal(c, in_turn) and bool(c.any())
print("SAME BITS")
"""


def test_no_room_for_k_block_sums():
    """On a device too full for the sums of K blocks side by side the call runs them in turn,
    with the same bits. In a process of its own, which has no workspace from earlier calls."""
    out = subprocess.run([sys.executable, "-c", NO_ROOM], capture_output=True, text=True, timeout=300)
    assert "SAME BITS" in out.stdout, out.stderr[-2000:]


@pytest.mark.parametrize("shape", [(300, 64, 333), (17, 20, 66), (2100, 132, 1429), (1, 4, 3)],
                         ids=lambda s: "x".join(map(str, s)))
def test_tf32_split_of_odd_rows(shape):
    """3xTF32 with rows of A that 16-byte accesses cannot split: the bits of the same matrix
    with zero columns up to a multiple of four, which they can."""
    import torch
    import flashgemm_b200 as fg
    M, N, K = shape
    K4 = (K + 3) // 4 * 4
    A, B = oracle.sgemm_inputs(M, N, K, seed=M + K)
    out = []
    for k in (K, K4):
        a, b = torch.zeros(M, k, device="cuda"), torch.zeros(k, N, device="cuda")
        a[:, :K], b[:K] = torch.from_numpy(A), torch.from_numpy(B)
        c = torch.full((M, N), 7.0, device="cuda")
        fg.sgemm_dev(c, a, b, M, N, k, algo="3xtf32")
        fg.sync()
        out.append(c.cpu().numpy())
    np.testing.assert_array_equal(out[0], out[1])
