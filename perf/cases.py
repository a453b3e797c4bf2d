"""The work that this library is timed on: GEMM chains, single GEMMs, grouped
plans and the serving loop, each through its public entry point.

A case names a kind and its sizes:

  chain   C = A_n ... A_1 B of one dtype (bf16, int8, f32 = split-precision 3xTF32,
          f32-ffma = plain FP32), by one of three callers: "dev" (weights in device
          memory handed over on each call), "registered" (weights prepared once and kept),
          "host" (the drop-in entry points on ordinary host arrays)
  sgemm   one FP32 GEMM, "ffma" (the reference's bits) or "3xtf32", on device memory, or
          through LibShalom_sgemm_mp on host arrays
  group   a plan of FP32 chains of mixed lengths and shapes, replayed through its graph
  serve   a burst of mixed requests on resident weights through the serving loop

Sizes are those of the benchmark, of the shape tables that the reference's test programs
time (repeated in tests/test_gpu_ref_shapes.py) and of the grouped and serving workloads'
distributions. INT8 stages between others have rows in multiples of 4 and BF16 ones in
multiples of 2, where the reference's result is defined.
"""
import math
import random

import numpy as np
import torch

import flashgemm_b200 as fg

# (N, K1, M1, M2, M3): multigemm/test/test_{f32,bf16,int8}_3.c:14-48
TABLE = [(65536, 288, 32, 24, 144), (16384, 1296, 144, 32, 192), (16384, 1728, 192, 32, 192),
         (4096, 4800, 192, 56, 336), (4096, 8400, 336, 56, 336), (50176, 288, 32, 16, 96),
         (12544, 864, 96, 24, 144), (12544, 1296, 144, 24, 144), (3136, 1296, 144, 32, 192),
         (3136, 1728, 192, 32, 192)]
# most work of a drawn case: that of the largest listed one of its kind
MOST_CHAIN = {"bf16": 7.8e10, "int8": 4.9e11, "f32": 2e10, "f32-ffma": 1e10}
MOST_SGEMM = 1.3e11
MOST_GROUP = 1.6e11
MOST_SERVE = 4e11


def listed():
    return [
        # the serving stream's smallest request: latency and the launch are all there is
        {"name": "chain-bf16-small", "kind": "chain", "dtype": "bf16", "how": "registered", "N": 64,
         "dims": "64,64,64"},
        # the benchmark's BF16 chain (a transformer-like MLP block and a projection)
        {"name": "chain-bf16-wide", "kind": "chain", "dtype": "bf16", "how": "dev", "N": 4096,
         "dims": "1024,4096,1024,1024"},
        # the benchmark's INT8 chain: the largest resident-weights call
        {"name": "chain-int8-wide", "kind": "chain", "dtype": "int8", "how": "registered", "N": 8192,
         "dims": "2048,4096,2048,4096,1024"},
        # the reference's table: convolution-like chains, wide activations on narrow stages
        {"name": "chain-bf16-table", "kind": "chain", "dtype": "bf16", "how": "dev", "N": 16384,
         "dims": "1296,144,32,192"},
        # the same table where the first stage is deep and there are few columns
        {"name": "chain-int8-table", "kind": "chain", "dtype": "int8", "how": "dev", "N": 4096,
         "dims": "4800,192,56,336"},
        # the same table in FP32, on the library's default algorithm
        {"name": "chain-f32-table", "kind": "chain", "dtype": "f32", "how": "dev", "N": 12544,
         "dims": "864,96,24,144"},
        # a drop-in caller of the reference: ordinary host arrays in, host array out
        {"name": "chain-bf16-host", "kind": "chain", "dtype": "bf16", "how": "host", "N": 12544,
         "dims": "1296,144,24,144"},
        # the benchmark's single FP32 GEMM
        {"name": "sgemm-1024", "kind": "sgemm", "algo": "ffma", "how": "dev", "M": 1024, "N": 1024,
         "K": 1024},
        # singlegemm's odd shape: ragged in every way, and K cut into blocks of 2048
        {"name": "sgemm-ragged", "kind": "sgemm", "algo": "ffma", "how": "dev", "M": 35, "N": 8457,
         "K": 2560},
        # singlegemm's largest shape
        {"name": "sgemm-large", "kind": "sgemm", "algo": "ffma", "how": "dev", "M": 1632, "N": 36548,
         "K": 1024},
        # a graph-replayed plan of FP32 chains, two tall-skinny ones among them
        {"name": "group-f32", "kind": "group", "chains": 24, "skinny": 2, "mix": 4321},
        # a burst of requests on resident weights
        {"name": "serve-burst", "kind": "serve", "requests": 48, "sets": 24, "mix": 777},
    ]


# ---------------------------------------------------------------- shapes

def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(max(step * round(v / step), lo), hi))


def _dims(case):
    return [int(x) for x in case["dims"].split(",")]


def _chain_flops(N, dims):
    return sum(2.0 * N * k * m for k, m in zip(dims, dims[1:]))


def _elt(dtype):
    return {"bf16": 2, "int8": 1}.get(dtype, 4)


def _group_specs(case):
    """Chain length U{2..5}, dims log-uniform on multiples of 16 in [64, 4096], columns in
    [64, 8192], and chains of 65536 columns with 64 x 64 weights; at most MOST_GROUP work."""
    rng = random.Random(case["mix"])
    out, left = [], MOST_GROUP
    for i in range(case["chains"] - case["skinny"]):
        while True:
            dims = [_log(rng, 64, 4096, 16) for _ in range(rng.randint(2, 5) + 1)]
            N = _log(rng, 64, 8192, 16)
            if _chain_flops(N, dims) <= max(left / 3, MOST_GROUP / 200):
                break
        left -= _chain_flops(N, dims)
        out.append((N, dims))
    for _ in range(case["skinny"]):
        out.append((65536, [64] * (rng.randint(2, 5) + 1)))
    rng.shuffle(out)
    return out


def _serve_specs(case):
    """Weight sets (length U{2..6}, dims log-uniform on multiples of 16 in [64, 4096], 50 %
    BF16 / 30 % INT8 / 20 % FP32) and requests (set, columns log-uniform in [64, 4096])."""
    rng = random.Random(case["mix"])
    sets = []
    for _ in range(case["sets"]):
        dt = rng.choices(["bf16", "int8", "f32"], [0.5, 0.3, 0.2])[0]
        sets.append((dt, [_log(rng, 64, 4096, 16) for _ in range(rng.randint(2, 6) + 1)]))
    reqs, left = [], MOST_SERVE
    for _ in range(case["requests"]):
        while True:
            i, N = rng.randrange(len(sets)), _log(rng, 64, 4096, 16)
            if _chain_flops(N, sets[i][1]) <= max(left / 4, MOST_SERVE / 400):
                break
        left -= _chain_flops(N, sets[i][1])
        reqs.append((i, N))
    return sets, reqs


def draw(rng):
    kind = rng.choices(["chain", "sgemm", "group", "serve"], [6, 4, 1, 1])[0]
    if kind == "group":
        return {"kind": "group", "chains": rng.randint(8, 24), "skinny": rng.randint(0, 2),
                "mix": rng.randrange(1 << 30)}
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(8, 48), "sets": rng.randint(8, 24),
                "mix": rng.randrange(1 << 30)}
    if kind == "sgemm":
        how = rng.choices(["dev", "host"], [4, 1])[0]
        algo = "ffma" if how == "host" else rng.choices(["ffma", "3xtf32"], [3, 1])[0]
        while True:
            M, N, K = _log(rng, 32, 32000), _log(rng, 16, 40000), _log(rng, 32, 8192)
            if rng.random() < 0.6:
                M, N, K = [max(16, 16 * round(x / 16)) for x in (M, N, K)]
            if algo == "3xtf32":
                N = 4 * max(4, round(N / 4))  # the entry point takes whole 16-byte rows
            most = MOST_SGEMM if how == "dev" else 2e10
            if 2.0 * M * N * K <= most and (how == "dev" or M * K + K * N + M * N <= 1 << 25):
                return {"kind": "sgemm", "algo": algo, "how": how, "M": M, "N": N, "K": K}
    dtype = rng.choices(["bf16", "int8", "f32", "f32-ffma"], [4, 3, 3, 1])[0]
    how = rng.choices(["dev", "registered", "host"], [2, 2, 1])[0]
    even = 4 if dtype == "int8" else 2
    while True:
        if rng.random() < 0.5:  # wide activations on narrow stages
            N = _log(rng, 3136, 65536)
            dims = [_log(rng, 288, 8400, even)] + [_log(rng, 16, 336, 4)
                                                   for _ in range(rng.randint(1, 3))]
        else:
            N = _log(rng, 64, 8192)
            dims = [_log(rng, 64, 4096, 16) for _ in range(rng.randint(2, 6) + 1)]
        if rng.random() < 0.7:
            N = max(16, 16 * round(N / 16))
        most = MOST_CHAIN[dtype] if how != "host" else 2e10
        if _chain_flops(N, dims) <= most and (how != "host" or N * max(dims) <= 1 << 25):
            break
    return {"kind": "chain", "dtype": dtype, "how": how, "N": N,
            "dims": ",".join(str(d) for d in dims)}


# ---------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _weight(dtype, m, k, g):
    if dtype == "int8":
        return torch.randint(-127, 128, (m, k), generator=g, device="cuda", dtype=torch.int8)
    a = torch.randn(m, k, generator=g, device="cuda") / math.sqrt(k)
    return a.to(torch.bfloat16) if dtype == "bf16" else a


def _activation(dtype, k, n, g):
    if dtype == "int8":
        return torch.randint(-127, 128, (k, n), generator=g, device="cuda", dtype=torch.int8)
    b = torch.randn(k, n, generator=g, device="cuda")
    return b.to(torch.bfloat16) if dtype == "bf16" else b


def _chain_inputs(dtype, N, dims, g):
    A = [_weight(dtype, m, k, g) for k, m in zip(dims, dims[1:])]
    return A, _activation(dtype, dims[0], N, g)


def _result(dtype, m, n):
    # rows that the reference leaves untouched (INT8, past the last whole four) stay zero
    return torch.zeros(m, n, device="cuda", dtype=torch.int32 if dtype == "int8" else torch.float32)


def _abi(t):
    """The tensor as the entry points take it: BF16 by its 16-bit patterns."""
    return t.view(torch.int16) if t.dtype == torch.bfloat16 else t


def _host(t, dtype):
    a = _abi(t).cpu().numpy()
    return a.view(np.uint16) if dtype == "bf16" else a


def _sgemm_inputs(case, g):
    A = torch.rand(case["M"], case["K"], generator=g, device="cuda") * 2 - 1
    B = torch.rand(case["K"], case["N"], generator=g, device="cuda") * 2 - 1
    return A, B


def _serve_inputs(case, g):
    sets, reqs = _serve_specs(case)
    A = [[_weight(dt, m, k, g) for k, m in zip(dims, dims[1:])] for dt, dims in sets]
    B = [_activation(sets[i][0], sets[i][1][0], N, g) for i, N in reqs]
    return sets, reqs, A, B


def prepare(case, seed):
    g = _gen(seed)
    if case["kind"] == "sgemm":
        A, B = _sgemm_inputs(case, g)
        C = torch.zeros(case["M"], case["N"], device="cuda")
        if case["how"] == "host":
            A, B, C = (np.ascontiguousarray(t.cpu().numpy()) for t in (A, B, C))
        return dict(case, A=A, B=B, C=C)
    if case["kind"] == "chain":
        dims, dtype = _dims(case), case["dtype"].split("-")[0]
        A, B = _chain_inputs(dtype, case["N"], dims, g)
        C = _result(dtype, dims[-1], case["N"])
        st = dict(case, dt=dtype, Ms=dims[1:], Ks=dims[:-1], C=C, B=_abi(B), A=[_abi(a) for a in A])
        if case["how"] == "registered":
            st["W"] = [fg.Weights(dtype, a) for a in st["A"]]
        elif case["how"] == "host":
            st["C"] = np.ascontiguousarray(C.cpu().numpy())
            b = _host(B, dtype)
            st["B"] = b.view(np.uint8) if dtype == "int8" else b
            st["args"] = []
            for a, m, k in zip(A, st["Ms"], st["Ks"]):
                st["args"] += [_host(a, dtype), m, k]
        return st
    if case["kind"] == "group":
        chains = []
        for N, dims in _group_specs(case):
            A, B = _chain_inputs("f32", N, dims, g)
            chains.append((_result("f32", dims[-1], N), B, N, [fg.Weights("f32", a) for a in A]))
        fg.set_f32_algo("3xtf32")
        return dict(case, chains=chains, plan=fg.Plan("f32", chains))
    sets, reqs, A, B = _serve_inputs(case, g)
    W = [[fg.Weights(dt, _abi(a)) for a in As] for (dt, _), As in zip(sets, A)]
    C = [_result(sets[i][0], sets[i][1][-1], N) for i, N in reqs]
    return dict(case, server=fg.Server(hbm_budget=16 << 30), C=C, W=W,
                reqs=[(sets[i][0], W[i], _abi(b), c) for (i, N), b, c in zip(reqs, B, C)])


# ---------------------------------------------------------------- one pass

def run(st):
    kind = st["kind"]
    if kind == "sgemm":
        if st["how"] == "host":
            fg.LibShalom_sgemm_mp(0, 0, st["C"], st["A"], st["B"], st["M"], st["N"], st["K"], check=True)
        else:
            fg.sgemm_dev(st["C"], st["A"], st["B"], st["M"], st["N"], st["K"], algo=st["algo"])
        return st["C"]
    if kind == "chain":
        if st["dt"] == "f32":
            fg.set_f32_algo("ffma" if st["dtype"] == "f32-ffma" else "3xtf32")
        if st["how"] == "registered":
            fg.chain_registered(st["dt"], st["C"], st["B"], st["N"], st["W"])
        elif st["how"] == "dev":
            fg.chain_dev(st["dt"], st["C"], st["B"], st["N"], st["A"], st["Ms"], st["Ks"])
        else:
            f = {"f32": fg.flashgemm_multi_f32f32f32, "bf16": fg.flashgemm_multi_bf16bf16f32,
                 "int8": fg.flashgemm_multi_int8uint8int32}[st["dt"]]
            f(st["C"], st["B"], st["N"], len(st["Ms"]), *st["args"], check=True)
        return st["C"]
    if kind == "group":
        st["plan"].launch(graph=True)
        return [c[0] for c in st["chains"]]
    fg.set_f32_algo("3xtf32")
    ids = [st["server"].submit(dt, W, b, c) for dt, W, b, c in st["reqs"]]
    for rid in ids:
        st["server"].wait(rid)
    return st["C"]


# ---------------------------------------------------------------- what a pass cannot do without

def _chain_work(dtype, N, dims):
    e = _elt(dtype)
    weights = sum(k * m for k, m in zip(dims, dims[1:])) * e
    return weights + e * dims[0] * N + 4 * dims[-1] * N, _chain_flops(N, dims)


def work(case):
    if case["kind"] == "sgemm":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 4 * (M * K + K * N + M * N), "flops": 2.0 * M * N * K}
    if case["kind"] == "chain":
        parts = [_chain_work(case["dtype"], case["N"], _dims(case))]
    elif case["kind"] == "group":
        parts = [_chain_work("f32", N, dims) for N, dims in _group_specs(case)]
    else:
        sets, reqs = _serve_specs(case)
        columns = [0] * len(sets)  # a set's weights are read once for all of its requests
        for i, N in reqs:
            columns[i] += N
        parts = [_chain_work(dt, n, dims) for (dt, dims), n in zip(sets, columns) if n]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


# ---------------------------------------------------------------- the same in 64 bits

def _permute(x, r):
    """The reference's hand-over between stages: each block of r rows x 32 columns is stored
    row by row and read back column by column of r (r = 2 for BF16, 4 for INT8); a last panel
    narrower than 32 columns and rows past the last whole block stay as they are."""
    m, n = (x.shape[0] // r) * r, (x.shape[1] // 32) * 32
    if m == 0 or n == 0:
        return x
    y = x.clone()
    p = x[:m, :n].reshape(m // r, r, n // 32, 32).permute(0, 2, 1, 3).reshape(m // r, n // 32, 32 * r)
    y[:m, :n] = p.reshape(m // r, n // 32, 32, r).permute(0, 3, 1, 2).reshape(m, n)
    return y


def _int8_stage(a, x):
    """Unsigned weights on signed activations; rows [12 floor(M/12), 4 floor(M/4)) pair weight
    quad s with activation quad max(s - 1, 0)."""
    M, K = a.shape
    w = a.view(torch.uint8).double()
    c = w @ x
    lo, hi = M // 12 * 12, M // 4 * 4
    if K % 4 == 0 and lo < hi:
        c[lo:hi] = w[lo:hi] @ torch.cat([x[:4], x[:K - 4]])
    return c


def _chain_exact(dtype, A, B):
    x = B.double()
    for i, a in enumerate(A):
        c = _int8_stage(a, x) if dtype == "int8" else a.double() @ x
        if i + 1 == len(A):
            if dtype == "int8":
                c[c.shape[0] // 4 * 4:] = 0
                return c.to(torch.int32)
            return c
        if dtype == "int8":
            x = _permute(c.clamp(-128, 127), 4)
        elif dtype == "bf16":
            x = _permute(c.to(torch.bfloat16).double(), 2)
        else:
            x = c


def exact(case, seed):
    g = _gen(seed)
    if case["kind"] == "sgemm":
        A, B = _sgemm_inputs(case, g)
        return A.double() @ B.double()
    if case["kind"] == "chain":
        dtype = case["dtype"].split("-")[0]
        return _chain_exact(dtype, *_chain_inputs(dtype, case["N"], _dims(case), g))
    if case["kind"] == "group":
        return [_chain_exact("f32", *_chain_inputs("f32", N, dims, g))
                for N, dims in _group_specs(case)]
    sets, reqs, A, B = _serve_inputs(case, g)
    return [_chain_exact(sets[i][0], A[i], b) for (i, N), b in zip(reqs, B)]
