"""Page-locked host operands: one launch reads all of them (used rows of W and H, S), small results are written straight to
host memory, larger calls run in chunks.  Against the CPU oracle (tests/helpers.py) and the byte counts."""
import numpy as np
import pytest
import torch

from helpers import assert_parity, random_coo
from sddmm_gpu_b200 import api

pytestmark = pytest.mark.gpu


def _pinned(a, offset=0):
    t = torch.empty(a.size + offset, dtype=torch.float32).pin_memory()[offset:].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


# K below and above the line for used rows only; nonzeros not a multiple of 4 or of an S tile; P small enough to be written
# through the mapping and larger; an S slice that is not 16-byte aligned (copied instead); W alone on the host
@pytest.mark.parametrize("K,nnz,s_offset", [(4, 997, 0), (28, 5001, 0), (32, 5003, 1), (36, 2049, 0), (100, 70001, 0), (256, 66003, 3)])
def test_mapped_operands(engine, K, nnz, s_offset):
    rng = np.random.default_rng(K)
    M, N = 1501, 1203
    rows, cols = random_coo(rng, M, N, nnz, empty_rows=[0, 1, 2, 700, M - 1])
    cols = cols - cols % 2          # odd columns are empty
    keep = np.ones(rows.size, bool)
    keep[1:] = (rows[1:] != rows[:-1]) | (cols[1:] != cols[:-1])
    rows, cols = rows[keep], cols[keep]
    W = rng.standard_normal((M, K)).astype(np.float32)
    H = rng.standard_normal((N, K)).astype(np.float32)
    vals = rng.standard_normal(rows.size).astype(np.float32)
    plan = engine.plan_coo(M, N, rows, cols, K)
    Wp, Hp, Sp = _pinned(W), _pinned(H), _pinned(vals, s_offset)
    for sv, sp in ((vals, Sp), (None, None)):
        P = torch.full((rows.size,), float("nan")).pin_memory()
        plan.execute(Wp, Hp, P, sp)
        assert_parity(P.numpy(), rows, cols, W, H, sv)
    up, down = plan.last_transfer_bytes()
    lines = (np.unique(rows).size + np.unique(cols).size) if K >= 32 else M + N
    assert (up, down) == (4 * K * lines, 4 * rows.size)
    P = torch.full((rows.size,), float("nan")).pin_memory()
    plan.execute(Wp, Hp.cuda(), P, Sp)           # H on the device
    assert_parity(P.numpy(), rows, cols, W, H, vals)
    Pd = torch.full((rows.size,), float("nan"), device="cuda")
    plan.execute(Wp, Hp, Pd)                      # P on the device
    assert_parity(Pd.cpu().numpy(), rows, cols, W, H)
    plan.close()


def test_chunked_call_keeps_its_kernel_time(engine):
    # 64 MB of W in two chunks; the time of each plan's last call is its own although the chunk events are shared
    rng = np.random.default_rng(0)
    M, N, K = 262144, 512, 64
    rows = np.sort(rng.integers(0, M, 200_001)).astype(np.int32)
    cols = rng.integers(0, N, rows.size).astype(np.int32)
    W, H = (rng.standard_normal((n, K)).astype(np.float32) for n in (M, N))
    Wp, Hp = _pinned(W), _pinned(H)
    plans = [engine.plan_coo(M, N, rows[:n], cols[:n], K) for n in (200_001, 150_000)]
    for plan in plans:
        P = torch.full((plan.nnz,), float("nan")).pin_memory()
        plan.execute(Wp, Hp, P)
        assert plan.last_kernel_name() == "gather (pipelined chunks)"
        assert_parity(P.numpy(), rows[:plan.nnz], cols[:plan.nnz], W, H)
    times = [plan.last_kernel_ms() for plan in plans]
    assert all(t > 0 for t in times) and times == [plan.last_kernel_ms() for plan in plans]
    for plan in plans:
        plan.close()


def test_chunks_taken_together_for_a_pageable_result(engine):
    # 168 MB of W are five chunks; with P in pageable memory four of them go together, then the last one
    rng = np.random.default_rng(1)
    M, N, K = 656_000, 300, 64
    rows = np.sort(rng.integers(0, M, 150_003)).astype(np.int32)
    cols = rng.integers(0, N, rows.size).astype(np.int32)
    W, H = (rng.standard_normal((n, K)).astype(np.float32) for n in (M, N))
    vals = rng.standard_normal(rows.size).astype(np.float32)
    plan = engine.plan_coo(M, N, rows, cols, K)
    Wp = _pinned(W)
    for operand in (W, Wp, W):
        P = np.full(rows.size, np.nan, np.float32)
        plan.execute(operand, H, P, vals)
        assert plan.last_kernel_name() == "gather (pipelined chunks)" and plan.last_kernel_ms() > 0
        assert_parity(P, rows, cols, W, H, vals)
        Pp = torch.full((rows.size,), float("nan")).pin_memory()       # chunk by chunk
        plan.execute(operand, H, Pp, vals)
        assert plan.last_kernel_ms() > 0 and np.array_equal(Pp.numpy(), P)
    plan.close()


def test_chunks_are_split_as_the_whole(engine):
    # 77 MB of W in two chunks of 0.6 M nonzeros, of a matrix of 1.2 M that is multiplied in two passes over the columns: the chunks as well,
    # so that P has the same bits wherever W is
    M, N, K, nnz = 50_003, 300_007, 384, 1_200_007
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    W, H = (torch.randn((n, K), generator=g, device="cuda") for n in (M, N))
    plan = engine.plan_coo(M, N, rows, cols, K)
    P, P_host = torch.full((nnz,), float("nan"), device="cuda"), torch.full((nnz,), float("nan")).pin_memory()
    n0 = engine.kernel_launches()
    plan.execute(W, H, P)
    assert engine.kernel_launches() - n0 == 2
    plan.execute(W.cpu().pin_memory(), H, P_host)
    assert plan.last_kernel_name() == "gather (pipelined chunks)" and plan.last_kernel_ms() > 0
    assert torch.equal(P.cpu(), P_host)
    plan.close()
