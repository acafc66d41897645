"""The calls whose speed matters: what a program that uses this library has it do, on one GPU.

A case names a call ("op"), the sparsity pattern it runs on and its sizes:

  op       sddmm   Plan.execute on a pattern planned before, operands on the GPU
           coo     Handle.sddmm_coo: no plan, a pattern that is used once
           replan  Handle.plan_coo, Plan.execute and Plan.close: a new pattern for every step (sampled minibatches)
           spmm    Plan.spmm, Y = P H (the product that follows SDDMM; also the gradient of SDDMM in W)
           fused   Plan.fused, Y = (S o W H^T) H, with or without P stored
           host    Plan.execute with W, H, S and P in page-locked host memory: the whole trip over PCIe
  pattern  uniform, words (documents x vocabulary), graph (R-MAT power law), attention (band + global rows and columns)
  dtype    storage of W and H: f32, or bf16 with FLAG_OPERANDS_BF16
  scaled   whether S values are given
  sync     the plain call, which waits for its result; otherwise FLAG_ASYNC on torch's current stream
"""
import math

import numpy as np
import torch

from sddmm_gpu_b200 import api, synth

# R-MAT quadrant probabilities of the benchmark's graphs; a row bit is 0 with A + B, a column bit with A + C
RMAT = (0.57, 0.19, 0.19, 0.05)


def _case(name, op, pattern, M, N, nnz, K, scaled=True, sync=False, dtype="f32", store_p=False, half_width=0, n_global=0):
    return dict(name=name, op=op, pattern=pattern, M=M, N=N, nnz=nnz, K=K, scaled=scaled, sync=sync, dtype=dtype,
                store_p=store_p, half_width=half_width, n_global=n_global)


def listed():
    return [
        # the smallest benchmark configuration: a call of some microseconds, its result awaited
        _case("uniform_4k_k32", "sddmm", "uniform", 4096, 4096, 16777, 32, sync=True),
        # documents x vocabulary (factorisation with a few thousand columns), the reference's own kind of input
        _case("words_12k_k256", "sddmm", "words", 12419, 1500, 746316, 256, sync=True),
        # a graph of a million vertices at an ordinary feature width
        _case("graph_1m_k128", "sddmm", "graph", 1 << 20, 1 << 20, 16085000, 128),
        # the headline benchmark: the largest graph, operands far beyond L2
        _case("graph_4m_k256", "sddmm", "graph", 1 << 22, 1 << 22, 96986616, 256),
        # sparse attention scores of one head: 64 K tokens, a band and global tokens
        _case("attention_64k_k64", "sddmm", "attention", 65536, 65536, 0, 64, half_width=256, n_global=80),
        # ragged sizes: M != N, no power of two anywhere, a row that is no multiple of 128 bytes, no S values
        _case("graph_ragged_k100", "sddmm", "graph", 300007, 250013, 4100001, 100, scaled=False),
        # one-shot call on a pattern that is not kept
        _case("coo_100k_k64", "coo", "graph", 100003, 100003, 1600000, 64),
        # a sampled neighbourhood: planned, used once, dropped -- every training step
        _case("replan_20k_k128", "replan", "graph", 20000, 50021, 400000, 128),
        # message passing with edge scores computed on the fly, edge scores not kept
        _case("fused_1m_k256", "fused", "graph", 1 << 20, 1 << 20, 16085000, 256),
        # aggregation / gradient: sparse values times features
        _case("spmm_250k_k64", "spmm", "graph", 250000, 250000, 6000003, 64),
        # everything in host memory, as the reference's callers have it
        _case("host_1m_k128", "host", "graph", 1 << 20, 1 << 20, 16085000, 128, sync=True),
        # features stored in bfloat16
        _case("bf16_1m_k256", "sddmm", "graph", 1 << 20, 1 << 20, 16085000, 256, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# feature widths: powers of two, the usual embedding sizes, and any multiple of four
WIDTHS = [32, 64, 64, 128, 128, 256, 256, 512, 48, 96, 100, 192, 200, 300, 384, 768]


def draw(rng):
    op = rng.choice(["sddmm"] * 9 + ["coo"] * 2 + ["replan"] * 2 + ["spmm"] * 3 + ["fused"] * 3 + ["host"])
    pattern = rng.choice(["graph", "graph", "graph", "uniform", "words", "attention"])
    K = rng.choice(WIDTHS) if rng.random() < 0.8 else 4 * rng.randint(4, 192)
    scaled, sync, dtype = rng.random() < 0.7, rng.random() < 0.4, "f32"
    half_width = n_global = 0
    if op == "host":
        pattern, sync = "graph", True
    if op in ("coo", "replan"):
        sync = True  # both wait by themselves or are called the plain way
    if op == "sddmm" and pattern == "graph" and rng.random() < 0.2:
        dtype, K = "bf16", rng.choice([256, 256, 512, 1024])
    if pattern == "attention":
        M = N = _log(rng, 1000, 50000)
        half_width = rng.randint(32, 256)
        n_global = rng.randint(0, 80)
        K = rng.choice([32, 64, 64, 96, 128])
        nnz = 0
    elif pattern == "words":
        M, N = _log(rng, 2000, 40000), _log(rng, 500, 4000)
        nnz = M * rng.randint(20, min(90, N // 10))
    elif pattern == "uniform":
        M, N = _log(rng, 500, 200000), _log(rng, 500, 200000)
        nnz = _log(rng, 1000, min(2000000, M * N // 10))
    else:
        M = _log(rng, 1000, 250000 if op in ("replan", "coo") else 1500000)
        N = max(1000, min(1500000, int(M * math.exp(rng.uniform(-1.2, 1.2)))))
        nnz = min(M, N) * rng.randint(4, 24) + rng.randint(0, 31)
    if op in ("spmm", "fused") and K > 512:
        K = 512
    if op == "host":
        K = min(K, 128)
    c = _case("", op, pattern, M, N, nnz, K, scaled=scaled, sync=sync, dtype=dtype,
              store_p=op == "fused" and rng.random() < 0.4, half_width=half_width, n_global=n_global)
    del c["name"]
    return c


# ---- inputs ---------------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _exactly(keys, nnz, g):
    """nnz of the (sorted, distinct) keys, those left out picked at random; sorted."""
    drop = keys.shape[0] - nnz
    if drop <= 0:
        return keys
    gone = torch.randperm(keys.shape[0], generator=g, device="cuda")[:drop]
    keep = torch.ones(keys.shape[0], dtype=torch.bool, device="cuda")
    keep[gone] = False
    return keys[keep]


def _uniform_keys(M, N, nnz, g):
    keys = torch.empty(0, dtype=torch.int64, device="cuda")
    while keys.shape[0] < nnz:
        more = torch.randint(0, M * N, (nnz + nnz // 16 + 64,), generator=g, device="cuda", dtype=torch.int64)
        keys = torch.unique(torch.cat([keys, more]))
    return _exactly(keys, nnz, g)


def _bits(n):
    return max(1, (n - 1).bit_length())


def _rmat_keys(M, N, nnz, g, chunk=1 << 24):
    """Distinct R-MAT cells of an M x N matrix (cells outside are drawn again)."""
    a, b, c, _ = RMAT
    br, bc = _bits(M), _bits(N)
    keys, left = torch.empty(0, dtype=torch.int64, device="cuda"), nnz + nnz // 24
    while keys.shape[0] < nnz:
        parts = [keys]
        while left > 0:
            n = min(left + left // 2, chunk)
            r = torch.zeros(n, dtype=torch.int64, device="cuda")
            col = torch.zeros(n, dtype=torch.int64, device="cuda")
            for i in range(max(br, bc)):
                u = torch.rand(n, generator=g, device="cuda")
                if i < br:
                    r = (r << 1) | (u >= a + b).to(torch.int64)
                if i < bc:
                    col = (col << 1) | (((u >= a) & (u < a + b)) | (u >= a + b + c)).to(torch.int64)
            inside = (r < M) & (col < N)
            k = (r * N + col)[inside][:left]
            left -= k.shape[0]
            parts.append(torch.unique(k))
        keys = torch.unique(torch.cat(parts))
        left = max(4096, 2 * (nnz - keys.shape[0]))
    return _exactly(keys, nnz, g)


def _pattern(case, seed):
    """(rows, cols) on the GPU, int32, row-sorted with ascending columns; S values."""
    M, N, nnz, g = case["M"], case["N"], case["nnz"], _gen(seed)
    if case["pattern"] == "words":
        p = synth.bag_of_words(M=M, N=N, nnz=nnz, K=4, seed=seed, device="cuda")
        return p["rows"], p["cols"], p["vals"]
    if case["pattern"] == "attention":
        # a model's mask is the same from step to step: the seed changes queries, keys and values only
        p = synth.attention_mask(M=M, half_width=case["half_width"], n_global=case["n_global"], K=4, device="cuda")
        return p["rows"], p["cols"], p["vals"]
    keys = (_uniform_keys if case["pattern"] == "uniform" else _rmat_keys)(M, N, nnz, g)
    rows = torch.div(keys, N, rounding_mode="floor").to(torch.int32)
    cols = (keys - rows.to(torch.int64) * N).to(torch.int32)
    if case["pattern"] == "uniform":
        vals = torch.ones(rows.shape[0], device="cuda")
    else:
        vals = torch.randn(rows.shape[0], generator=g, device="cuda")
    return rows.contiguous(), cols.contiguous(), vals


def _operands(case, seed):
    g = _gen(seed + 1)
    shapes = (case["M"], case["K"]), (case["N"], case["K"])
    if case["pattern"] in ("uniform", "words"):
        return [torch.rand(s, generator=g, device="cuda") for s in shapes]
    sigma = 1.0 if case["pattern"] == "attention" else 0.1
    return [torch.randn(s, generator=g, device="cuda").mul_(sigma) for s in shapes]


_handles = []


def _handle():
    """One engine handle for the process, as a program keeps it."""
    if not _handles:
        _handles.append(api.Handle(0))
    return _handles[0]


def prepare(case, seed):
    op = case["op"]
    rows, cols, vals = _pattern(case, seed)
    W, H = _operands(case, seed)
    nnz = rows.shape[0]
    s = dict(op=op, M=case["M"], N=case["N"], K=case["K"], rows=rows, cols=cols, W=W, H=H, handle=_handle(),
             flags=0 if case["sync"] else api.FLAG_ASYNC, S=vals if case["scaled"] else None)
    if case["dtype"] == "bf16":
        s["W"], s["H"] = W.to(torch.bfloat16), H.to(torch.bfloat16)
        s["flags"] |= api.FLAG_OPERANDS_BF16
    if op in ("spmm", "fused"):
        s["Y"] = torch.zeros((case["M"], case["K"]), device="cuda")
    if op != "spmm" and (op != "fused" or case["store_p"]):
        s["P"] = torch.zeros(nnz, device="cuda")
    if op == "host":
        for k in ("W", "H", "S", "P"):
            if s[k] is not None:
                s[k] = s[k].cpu().pin_memory()
    if op not in ("coo", "replan"):
        s["plan"] = s["handle"].plan_coo(case["M"], case["N"], rows, cols, case["K"])
    return s


def run(s):
    op = s["op"]
    if op in ("sddmm", "host"):
        s["plan"].execute(s["W"], s["H"], s["P"], s["S"], s["flags"])
        return s["P"]
    if op == "coo":
        s["handle"].sddmm_coo(s["M"], s["N"], s["rows"], s["cols"], s["W"], s["H"], s["K"], s["P"], s["S"])
        return s["P"]
    if op == "replan":
        plan = s["handle"].plan_coo(s["M"], s["N"], s["rows"], s["cols"], s["K"])
        plan.execute(s["W"], s["H"], s["P"], s["S"], s["flags"])
        plan.close()
        return s["P"]
    if op == "spmm":
        s["plan"].spmm(s["H"], s["Y"], s["S"], s["flags"])
        return s["Y"]
    s["plan"].fused(s["W"], s["H"], s["Y"], s["S"], s.get("P"), s["flags"])
    return [s["Y"], s["P"]] if "P" in s else s["Y"]


# ---- the least work of a pass -----------------------------------------------------------------------------------

def _rmat_touched(n, nnz, p0):
    """Expected number of the n lines that hold one of nnz R-MAT cells; p0: probability of a zero bit."""
    bits = _bits(n)
    ids = np.arange(n, dtype=np.int64)
    ones = np.zeros(n, dtype=np.int64)
    for i in range(bits):
        ones += (ids >> i) & 1
    p = p0 ** (bits - ones) * (1.0 - p0) ** ones
    return float(np.sum(1.0 - np.exp(-nnz * p / p.sum())))


def work(case):
    M, N, nnz, K, op = case["M"], case["N"], case["nnz"], case["K"], case["op"]
    m, n = float(M), float(N)  # rows of W and of H that some nonzero touches
    if case["pattern"] == "graph":
        m, n = _rmat_touched(M, nnz, RMAT[0] + RMAT[1]), _rmat_touched(N, nnz, RMAT[0] + RMAT[2])
    elif case["pattern"] == "uniform":
        m, n = M * (1.0 - math.exp(-nnz / M)), N * (1.0 - math.exp(-nnz / N))
    elif case["pattern"] == "attention":
        h, g = case["half_width"], case["n_global"]
        h = min(h, M - 1)
        nnz = M * (2 * h + 1) - h * (h + 1) + 2 * g * M - g * g - 2 * g * (2 * h + 1) + g
    row = K * (2 if case["dtype"] == "bf16" else 4)
    values = 4 * nnz if case["scaled"] else 0
    flops = 2.0 * nnz * K
    if op == "spmm":
        total = row * n + 4 * K * M + 4 * nnz + values + 4 * (M + 1)
    elif op == "fused":
        total = row * (m + n) + 4 * K * M + 4 * nnz + values + (4 * nnz if case["store_p"] else 0) + 4 * (M + 1)
        flops *= 2
    else:  # W and H rows, a column index and a P store per nonzero, S values, and a row index or pointer
        total = row * (m + n) + 8 * nnz + values + (4 * nnz if op in ("coo", "replan") else 4 * (M + 1))
    return {"bytes": float(total), "flops": float(flops)}


def tolerance(case):
    # 32-bit products and sums of at most K (P) or of K and a row's length (Y) terms; bfloat16 operands are given as
    # such and their products are exact in 32 bits
    return {"rel": 1e-5}
