"""FP32 (3xTF32) chains whose intermediates stay in tensor memory: the same bits as one
launch per stage, at the edges of the tiles (rows, k, columns, several row tiles of the
last stage, several blocks per CTA), in one launch on registered weights."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

# N, K_1, (M_1, ..., M_n)
SHAPES = [
    (128, 96, (96, 24, 144)),            # the reference's widths, one block
    (4, 66, (2, 2, 1)),                  # the smallest dimensions (a smaller K_1: panel-resident)
    (132, 98, (16, 18, 17)),             # k and rows past a multiple of 16, 8 and 2
    (260, 72, (48, 48, 48)),             # the half-SM build's widest
    (388, 66, (50, 32, 400)),            # the full build, last stage in several tiles
    (1000, 514, (144, 32, 192)),         # the widest intermediate
    (640, 2050, (144, 144)),             # chunks of three k-blocks
    (900, 864, (130,)),                  # one stage
    (300, 72, (66, 8, 70, 64, 10, 64, 36, 20)),   # eight stages
    (40004, 96, (32, 16, 96)),           # more blocks than CTAs, half-SM build
    (20480, 70, (96, 20, 30)),           # the same, full build
]


@pytest.mark.parametrize("shape", SHAPES, ids=[f"n{n}_k{k}_" + "-".join(map(str, m)) for n, k, m in SHAPES])
def test_column_chain_same_bits_as_stages(shape):
    import torch
    import flashgemm_b200 as fg
    N, K1, Ms = shape
    Ms = list(Ms)
    B, As, Ks = oracle.chain_inputs("f32", N, K1, Ms, seed=N + K1)
    W = [fg.Weights("f32", a) for a in As]
    b = torch.from_numpy(B).cuda()
    fg.set_f32_algo("3xtf32")

    def run():
        c = torch.full((Ms[-1], N), 7.0, device="cuda")
        before = fg.kernel_launches()
        fg.chain_registered("f32", c, b, N, W)
        fg.sync()
        return c.cpu().numpy(), fg.kernel_launches() - before

    got, launches = run()
    fg.set_chain_mode("per_gemm")
    try:
        want, _ = run()
    finally:
        fg.set_chain_mode("fused")
    assert launches == 1
    np.testing.assert_array_equal(got, want)
    for w in W:
        w.release()


@pytest.mark.parametrize("N", [1001, 5120])
def test_column_chain_unregistered_weights_and_odd_columns(N):
    import torch
    import flashgemm_b200 as fg
    Ms = [96, 24, 144]
    B, As, Ks = oracle.chain_inputs("f32", N, 866, Ms, seed=N)
    b, a = torch.from_numpy(B).cuda(), [torch.from_numpy(x).cuda() for x in As]
    fg.set_f32_algo("3xtf32")
    out = []
    for mode in ("fused", "per_gemm"):
        fg.set_chain_mode(mode)
        try:
            c = torch.zeros(Ms[-1], N, device="cuda")
            fg.chain_dev("f32", c, b, N, a, Ms, Ks)
            fg.sync()
        finally:
            fg.set_chain_mode("fused")
        out.append(c.cpu().numpy())
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("N", [1001, 5120])
def test_column_chain_unregistered_weights_is_two_launches(N):
    """The weights' split and the chain, where one launch per stage takes four."""
    import torch
    import flashgemm_b200 as fg
    Ms = [96, 24, 144]
    B, As, Ks = oracle.chain_inputs("f32", N, 866, Ms, seed=N)
    b, a = torch.from_numpy(B).cuda(), [torch.from_numpy(x).cuda() for x in As]
    c = torch.zeros(Ms[-1], N, device="cuda")
    fg.set_f32_algo("3xtf32")
    counts = []
    for mode in ("fused", "per_gemm"):
        fg.set_chain_mode(mode)
        try:
            before = fg.kernel_launches()
            fg.chain_dev("f32", c, b, N, a, Ms, Ks)
            fg.sync()
            counts.append(fg.kernel_launches() - before)
        finally:
            fg.set_chain_mode("fused")
    assert counts == [2, 4]


@pytest.mark.parametrize("shape", [(300, 98, (16, 18, 17)), (300, 514, (144, 32, 192)), (300, 98, (50, 32, 400))],
                         ids=["half-sm", "16-deep", "tiles"])
def test_bad_values_as_per_stage(shape):
    """Infinities, NaN and sums past the largest FP32 in B and in the weights: the same bits,
    or NaN, as one launch per stage, and every other column stays finite."""
    import torch
    import flashgemm_b200 as fg
    N, K1, Ms = shape
    Ms = list(Ms)
    B, As, Ks = oracle.chain_inputs("f32", N, K1, Ms, seed=K1)
    B, As = np.array(B), [np.array(a) for a in As]
    B[5, 40], B[K1 - 1, 131], B[7, 250] = np.inf, np.nan, 3.4e38
    fg.set_f32_algo("3xtf32")
    b = torch.from_numpy(B).cuda()

    def run(weights):
        out = []
        W = [fg.Weights("f32", a) for a in weights]
        for mode in ("fused", "per_gemm"):
            fg.set_chain_mode(mode)
            try:
                c = torch.zeros(Ms[-1], N, device="cuda")
                before = fg.kernel_launches()
                fg.chain_registered("f32", c, b, N, W)
                fg.sync()
                launches = fg.kernel_launches() - before
            finally:
                fg.set_chain_mode("fused")
            assert (launches == 1) == (mode == "fused")
            out.append(c.cpu().numpy())
        for w in W:
            w.release()
        np.testing.assert_array_equal(out[0], out[1])  # NaN equal to NaN
        return out[0]

    got = run(As)
    assert np.isfinite(np.delete(got, [40, 131, 250], axis=1)).all()
    assert not np.isfinite(got[:, [40, 131]]).any()
    As[-1][3, 2] = np.inf
    got = run(As)
    assert not np.isfinite(got[3]).any() and np.isfinite(np.delete(got, [40, 131, 250], axis=1)[4:]).all()
