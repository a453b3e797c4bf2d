"""Narrow BF16 / INT8 chains at the edges of their kernel's tiles: rows around the 16-row
groups and the two row tiles of the last stage, columns around the
32-column panels and the 128-column blocks, more blocks than SMs (two CTAs per SM), and
infinities and NaN in one column, which must not reach another. The per-GEMM path computes
the same products in the same order: the results are equal bit for bit."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SHAPES = [
    # N, K1, Ms
    (1, 16, [16, 4]),
    (31, 40, [2, 17]),
    (33, 130, [14, 34, 129]),            # last stage two tiles of 80 rows
    (127, 64, [132, 136]),               # INT8 tail rows across the tile edge
    (160, 200, [140, 254, 256]),
    (129, 4100, [18, 30, 257]),          # a last k-block of 4; last stage three tiles
    (19100, 96, [48, 24, 20]),           # 150 blocks
    (19000, 72, [250, 130, 200]),        # 149 blocks too wide for two CTAs per SM
    (300, 64, [8] * 8),                  # the most stages
]


@pytest.fixture(scope="module", autouse=True)
def fg():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import flashgemm_b200 as fg
    fg.lib()
    fg.set_semantics("ref")
    fg.set_chain_mode("fused")
    fg.set_narrow("always")
    fg.flashgemm_set_thread_num(1)
    yield fg
    fg.set_semantics("ref")
    fg.set_chain_mode("fused")
    fg.set_narrow("auto")


def _both(fg, dt, B, As, N, Ms, Ks):
    fn = {"bf16": fg.flashgemm_multi_bf16bf16f32, "int8": fg.flashgemm_multi_int8uint8int32}[dt]
    trip = [x for t in zip(As, Ms, Ks) for x in t]
    out = []
    for mode in ("fused", "per_gemm"):
        C = np.zeros((Ms[-1], N), np.int32 if dt == "int8" else np.float32)
        fg.set_chain_mode(mode)
        try:
            launches = fg.kernel_launches()
            fn(C, B, N, len(As), *trip, check=True)
            launches = fg.kernel_launches() - launches
        finally:
            fg.set_chain_mode("fused")
        out.append((C, launches))
    return out


@pytest.mark.parametrize("sem", ["ref", "math"])
@pytest.mark.parametrize("dt", ["int8", "bf16"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"n{s[0]}_k{s[1]}_" + "-".join(map(str, s[2])))
def test_edges_equal_per_gemm(fg, dt, sem, shape):
    N, K1, Ms = shape
    B, As, Ks = oracle.chain_inputs(dt, N, K1, Ms, seed=7 * N + K1)
    fg.set_semantics(sem)
    try:
        (C, _), (ref, _) = _both(fg, dt, B, As, N, Ms, Ks)
    finally:
        fg.set_semantics("ref")
    assert np.array_equal(C, ref)


@pytest.mark.parametrize("value", [0x7F80, 0x7FC0], ids=["inf", "nan"])
def test_one_bad_column_stays_alone(fg, value):
    N, K1, Ms = 96, 72, [20, 34, 40]
    B, As, Ks = oracle.chain_inputs("bf16", N, K1, Ms, seed=3)
    B = np.array(B)
    B.view(np.uint16)[5, 40] = value
    fg.set_semantics("math")  # no panel permutation: a column of B is a column of C
    try:
        (C, _), (ref, _) = _both(fg, "bf16", B, As, N, Ms, Ks)
    finally:
        fg.set_semantics("ref")
    assert np.array_equal(C, ref, equal_nan=True)
    assert np.isfinite(np.delete(C, 40, axis=1)).all() and not np.isfinite(C[:, 40]).any()


TRACED = """
import glob, os, sys
sys.path.insert(0, sys.argv[1])
import conftest, oracle
import flashgemm_b200 as fg
import test_gpu_narrow_edges as t
fg.set_chain_mode("fused")
fg.set_narrow("always")
traces = lambda kind: len(glob.glob(os.path.join(os.environ["FG_TRACE_DIR"], kind + "_trace_*.csv")))
for N, K1, Ms in t.SHAPES:
    for dt in ("bf16", "int8"):
        B, As, Ks = oracle.chain_inputs(dt, N, K1, Ms, seed=1)
        for sem in ("ref", "math"):
            fg.set_semantics(sem)
            before = traces("narrow")
            t._both(fg, dt, B, As, N, Ms, Ks)
            assert traces("narrow") > before, (dt, sem, N, K1, Ms)
assert traces("chain") == 0
print("ALL NARROW")
"""


def test_edges_run_on_the_narrow_kernel(tmp_path):
    """Every shape above, in both types and semantics, leaves the narrow kernel's timeline
    and none of the fused kernel's."""
    env = dict(os.environ, FG_TRACE_DIR=str(tmp_path))
    out = subprocess.run([sys.executable, "-c", TRACED, os.path.dirname(os.path.abspath(__file__))],
                         capture_output=True, text=True, timeout=300, env=env)
    assert "ALL NARROW" in out.stdout, out.stderr[-2000:]
