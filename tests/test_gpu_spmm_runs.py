"""SpMM and the fused form at the run boundaries of csrc/spmm.cu: rows that end exactly where a run ends, that cross one
boundary, that span a few runs, exactly sixteen and seventeen and hundreds, a row that begins in
the run where a row of seventeen ends, the same with blocks of runs (one and two groups of parts), stretches of empty rows, repeated calls (the counters are left at zero),
and every lane shape's first and last K.

Tolerance: as tests/test_gpu_spmm.py (1e-4 of the sum of magnitudes per entry of Y, against float64)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TOL = 1e-4


def _rows_of_lengths(rng, lengths, N):
    rows = np.repeat(np.arange(len(lengths)), lengths)
    cols = np.concatenate([np.sort(rng.choice(N, n, replace=False)) for n in lengths]) if rows.size else rows
    return rows.astype(np.int32), cols.astype(np.int32)


@pytest.mark.parametrize("K", [4, 16, 20, 32, 36, 48, 52, 64, 68, 96, 100, 128, 132, 192, 196, 256, 260, 384, 388, 512, 516, 640,
                               644, 768, 772, 896, 900, 1024])
def test_run_boundaries(engine, K):
    rng = np.random.default_rng(K)
    N = 6000
    # runs are 8 or 16 nonzeros at this size (4 where sets are four lanes)
    lengths = [16, 16, 0, 0, 32, 8, 8, 15, 2, 1, 1, 1, 0, 70, 250, 5000, 3, 0, 0, 0, 16, 129, 6000, 0]
    lengths = [6, 257, 9, 40, 272, 264, 140] + lengths   # row 1: 17 runs of 16, row 3 begins where it has ended
    lengths += [(-sum(lengths)) % 16 + 8, 4, 65, 129, 3, 60, 124, 4,
                8 + 16 * 15, 17 * 16, 5, 2]
    rows, cols = _rows_of_lengths(rng, lengths, N)
    M = len(lengths)
    vals = rng.standard_normal(rows.shape[0]).astype(np.float32)
    W = rng.standard_normal((M, K)).astype(np.float32)
    H = rng.standard_normal((N, K)).astype(np.float32)
    plan = engine.plan_coo(M, N, rows, cols, K)
    for pv in (vals, None):
        Y = np.full((M, K), np.nan, np.float32)
        plan.spmm(H, Y, pv)
        ref, A = oracle.cpu.spmm_f64(rows, cols, H, M, pv)
        assert np.all(np.abs(Y - ref) <= TOL * np.maximum(np.abs(ref), A) + 1e-30)
    Y, Y2, P = np.full((M, K), np.nan, np.float32), np.full((M, K), np.nan, np.float32), np.full(rows.shape[0], np.nan, np.float32)
    plan.fused(W, H, Y, vals, P)
    P64, A_p = oracle.cpu.sddmm_coo_f64(rows, cols, W, H, vals)
    assert np.all(np.abs(P - P64) <= TOL * np.maximum(np.abs(P64), A_p))
    ref, A = oracle.cpu.spmm_f64(rows, cols, H, M, P64.astype(np.float32))
    _, A_from_p = oracle.cpu.spmm_f64(rows, cols, H, M, A_p)   # an error of 1e-4 A_p in p moves Y by up to that times |H|
    assert np.all(np.abs(Y - ref) <= TOL * (np.maximum(np.abs(ref), A) + A_from_p) + 1e-30)
    for _ in range(3):
        Y2.fill(np.nan)
        plan.fused(W, H, Y2, vals)
        assert np.array_equal(Y, Y2)
    plan.close()


@pytest.mark.parametrize("K", [196, 200, 252, 256])
def test_tails_in_scratch(engine, K):
    # a million nonzeros (K = 256: 300,000) and more leave the tails of runs in scratch, K = 256 has other blocks below 85,000; whole numbers: exact sums, on both sides of the lines
    import torch
    N, M = 5_003, 60_001
    g = torch.Generator(device="cuda").manual_seed(K)
    H = torch.randint(-1, 2, (N, K), generator=g, device="cuda").float()
    for nnz in (84_999, 85_000, 299_999, 300_000, 999_999, 1_000_000, 1_300_007):
        rows = torch.sort((torch.rand(nnz, generator=g, device="cuda") ** 4 * M).to(torch.int32).clamp_(max=M - 1)).values   # rows of many blocks and of a few nonzeros, and none
        cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
        vals = torch.randint(-1, 2, (nnz,), generator=g, device="cuda").float()
        plan = engine.plan_coo(M, N, rows, cols, K)
        for pv in (vals, None):
            Y = torch.full((M, K), float("nan"), device="cuda")
            plan.spmm(H, Y, pv)
            ref = torch.zeros((M, K), device="cuda", dtype=torch.float64)
            for a in range(0, nnz, 200_000):
                part = H[cols[a:a + 200_000].long()].double()
                ref.index_add_(0, rows[a:a + 200_000].long(), part if pv is None else part * pv[a:a + 200_000, None].double())
            assert float(ref.abs().max()) < 2 ** 22 and torch.equal(Y.double(), ref)
        plan.close()


@pytest.mark.parametrize("K", [16, 32, 64, 96, 160, 192, 200, 256, 320, 384, 512, 768, 1024])
def test_block_boundaries(engine, K):
    # A block holds 8 to 64 runs of 8, 16 or 24 nonzeros (K = 16: of 4).  Rows that begin and end at multiples of 8 and 64 and one beside them, rows of a block and of
    # 16 and 17 blocks, many short rows in a run, rows that a block has only the end of; small whole numbers, so that every sum is exact.
    rng = np.random.default_rng(K)
    N = 17 * 1536 + 9
    lengths = [64, 64, 1, 63, 8, 56, 512, 7, 1, 504, 512 + 1, 511, 0, 1024, 8, 8, 48] + [1] * 32 + [2] * 16 + [16 * 64, 17 * 64, 16 * 192, 17 * 192, 16 * 512, 17 * 512 - 1, 1, 17 * 1536, 5, 3]
    lengths += [int(n) for n in rng.choice([8, 16, 24, 64, 128, 192, 256, 384, 512, 768], 60)]
    rows, cols = _rows_of_lengths(rng, lengths, N)
    M = len(lengths)
    vals = rng.integers(-1, 2, rows.shape[0]).astype(np.float32)
    W, H = rng.integers(-1, 2, (M, K)).astype(np.float32), rng.integers(-1, 2, (N, K)).astype(np.float32)
    P = np.einsum("ij,ij->i", W[rows], H[cols]) * vals   # at most K
    plan = engine.plan_coo(M, N, rows, cols, K)
    for weights, call in ((vals, lambda Y, p: plan.spmm(H, Y, vals)), (P, lambda Y, p: plan.fused(W, H, Y, vals, p))):
        ref, ends = np.zeros((M, K)), np.concatenate([[0], np.cumsum(lengths)])
        for r in range(M):
            ref[r] = weights[ends[r]:ends[r + 1]].astype(np.float64) @ H[cols[ends[r]:ends[r + 1]]]
        assert np.abs(ref).max() < 2 ** 20   # (random signs: partial sums are far from 2^24)
        for _ in range(2):   # (the counters are left at zero)
            Y, p = np.full((M, K), np.nan, np.float32), np.full(rows.shape[0], np.nan, np.float32)
            call(Y, p)
            assert np.array_equal(Y, ref.astype(np.float32))
            assert weights is vals or np.array_equal(p, P)
    plan.close()


@pytest.mark.parametrize("K", [4, 32, 36, 64, 96, 100, 128, 192, 252, 256, 384, 512, 640, 1024])
def test_last_nonzero_infinite(engine, K):
    # positive operands: the last row is +Inf everywhere, all other rows are finite; the matrix ends inside a step of every
    # shape, and inside a warp's last sets
    rng = np.random.default_rng(K)
    M, N = 40, 50
    for nnz in (1, 3, 5, 121, 1001):
        cells = np.sort(rng.choice((M - 1) * N, nnz - 1, replace=False))
        rows, cols = np.append(cells // N, M - 1).astype(np.int32), np.append(cells % N, 3).astype(np.int32)
        W, H = rng.random((M, K), dtype=np.float32) + 1, rng.random((N, K), dtype=np.float32) + 1
        vals = rng.random(nnz, dtype=np.float32) + 1
        infinite = vals.copy()
        infinite[-1] = np.inf
        W_inf = W.copy()
        W_inf[-1, K // 2] = np.inf
        plan = engine.plan_coo(M, N, rows, cols, K)
        for call, weights in ((lambda Y: plan.spmm(H, Y, infinite), vals),
                              (lambda Y: plan.fused(W, H, Y, infinite), None), (lambda Y: plan.fused(W_inf, H, Y, vals), None)):
            Y = np.full((M, K), np.nan, np.float32)
            call(Y)
            assert np.all(Y[-1] == np.inf)
            if weights is None:
                weights = oracle.cpu.sddmm_coo_f64(rows, cols, W, H, vals)[0].astype(np.float32)
            ref, A = oracle.cpu.spmm_f64(rows[:-1], cols[:-1], H, M, weights[:-1])
            # all terms are positive: an error of 1e-4 in each weight is one of 1e-4 in the sum
            assert np.all(np.abs(Y[:-1] - ref[:-1]) <= 2 * TOL * A[:-1])
        plan.close()


@pytest.mark.parametrize("K", [4, 16, 20, 32, 36, 48, 60, 64, 68, 96, 100, 128, 160, 192, 200, 256, 320, 384, 512, 640, 768, 896, 1024])
def test_fused_on_w(engine, K):
    # Y on the memory of W: rows of a few nonzeros and of many blocks, at the borders of runs, the same bits as with Y elsewhere
    import torch
    M, N = 3_001, 2_003
    g = torch.Generator(device="cuda").manual_seed(K)
    for nnz in (2_999, 60_007, 400_009):
        rows = torch.sort((torch.rand(nnz, generator=g, device="cuda") ** 4 * M).to(torch.int32).clamp_(max=M - 1)).values   # (and rows without any)
        cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
        W, H, S = (torch.randn(n, generator=g, device="cuda") for n in ((M, K), (N, K), (nnz,)))
        plan = engine.plan_coo(M, N, rows, cols, K)
        Y, P = torch.full((M, K), float("nan"), device="cuda"), torch.full((nnz,), float("nan"), device="cuda")
        plan.fused(W, H, Y, S, P)
        for _ in range(3):
            WY, P2 = W.clone(), torch.full((nnz,), float("nan"), device="cuda")
            plan.fused(WY, H, WY, S, P2)
            assert torch.equal(WY, Y) and torch.equal(P2, P)
            WY = W.clone()
            plan.fused(WY, H, WY, S)
            assert torch.equal(WY, Y)
        plan.close()


@pytest.mark.parametrize("K", [388, 512, 644, 768])
def test_weights_of_fused_as_sddmm(engine, K):
    # the same lanes hold the same pieces as in the gather kernel at these K, two sums a lane: P comes out with the same bits
    import torch
    M, N, nnz = 900, 1_100, 30_001
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    W, H, S = (torch.randn(n, generator=g, device="cuda") for n in ((M, K), (N, K), (nnz,)))
    plan = engine.plan_coo(M, N, rows, cols, K)
    P, P_fused, Y = torch.empty(nnz, device="cuda"), torch.full((nnz,), float("nan"), device="cuda"), torch.empty((M, K), device="cuda")
    plan.execute(W, H, P, S)
    plan.fused(W, H, Y, S, P_fused)
    plan.close()
    assert torch.equal(P, P_fused)


@pytest.mark.parametrize("K,N", [(448, 503_000), (512, 831_000), (900, 251_000)])
def test_long_rows_in_passes(engine, K, N):
    # a large H, long rows: passes over part of the columns (the last one of 64, 128 and 132), a row of many runs, rows without nonzeros
    import torch
    M, nnz = 7_013, 1_000_003
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = (torch.rand(nnz, generator=g, device="cuda") ** 3 * M).to(torch.int64).clamp_(max=M - 1)
    rows = torch.sort(torch.where(rows % 7 == 3, 0, rows)).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    H, vals = torch.randn((N, K), generator=g, device="cuda"), torch.randn(nnz, generator=g, device="cuda")
    plan = engine.plan_coo(M, N, rows, cols, K)
    for pv in (vals, None):
        n0 = engine.kernel_launches()
        Y = torch.full((M, K), float("nan"), device="cuda")
        plan.spmm(H, Y, pv)
        assert plan.last_kernel_ms() > 0 and engine.kernel_launches() - n0 == -(-K // 192)
        ref, A = (torch.zeros((M, K), device="cuda", dtype=torch.float64) for _ in range(2))
        for a in range(0, nnz, 100_000):
            t = H[cols[a:a + 100_000].long()].double()
            if pv is not None:
                t *= pv[a:a + 100_000, None].double()
            ref.index_add_(0, rows[a:a + 100_000].long(), t)
            A.index_add_(0, rows[a:a + 100_000].long(), t.abs())
        assert bool(((Y.double() - ref).abs() <= TOL * A).all())
        again = torch.full((M, K), float("nan"), device="cuda")
        plan.spmm(H, again, pv)
        assert torch.equal(Y, again)
    plan.close()


@pytest.mark.parametrize("K,M,n,block,chain", [(192, 11_400, 700, 2, 80), (200, 11_400, 700, 4, 80), (64, 40_000, 700, 4, 80), (576, 3_550, 80, 1, 32)])
def test_rounding_of_long_rows(engine, K, M, n, block, chain):
    # Rows of n positive terms, all of them as large on average.  A run adds at most `chain` times to a row's sum one after the other, `block`
    # nonzeros at a time, so the row is p = n / (chain block) such chains.  With an error of 2^-24 / sqrt(3) rms for every rounding, relative to the
    # partial sum: chain / 3 p from the chains, p / 3 from adding them up, 1 for the products.
    import torch
    N = 20_000
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.arange(M, device="cuda", dtype=torch.int32).repeat_interleave(n)
    cols = torch.randint(0, N, (M, n), generator=g, device="cuda").sort(dim=1).values
    H, vals = torch.rand((N, K), generator=g, device="cuda"), torch.rand((M, n), generator=g, device="cuda")
    plan = engine.plan_coo(M, N, rows, cols.flatten().to(torch.int32), K)
    Y = torch.full((M, K), float("nan"), device="cuda")
    plan.spmm(H, Y, vals.flatten())
    plan.close()
    square = 0.0
    for a in range(0, M, 200):
        ref = torch.einsum("mn,mnk->mk", vals[a:a + 200].double(), H[cols[a:a + 200]].double())
        square += float(((Y[a:a + 200].double() - ref) / ref).square().sum())
    p = n / (chain * block)
    assert (square / (M * K)) ** 0.5 <= 2.0 ** -24 / 3 ** 0.5 * (chain / (3 * p) + p / 3 + 1) ** 0.5


@pytest.mark.parametrize("fused,K,M,n,block,chain", [(False, 48, 550, 700, 2, 6), (True, 48, 550, 700, 2, 6), (True, 160, 550, 700, 1, 24), (False, 200, 2_000, 700, 4, 50), (True, 256, 9_300, 700, 4, 40),
                                                       (True, 512, 2_800, 700, 2, 48), (True, 96, 300_000, 100, 2, 50), (True, 32, 40_000, 700, 2, 76)])
def test_rounding_of_parts(engine, fused, K, M, n, block, chain):
    # As above, the fused form too (W picks a column of ones of H: the weights are S).  The p parts of a row are added eight at a time and the sums of eight one after the other, and a row
    # goes over to the next block: 1 more.  A rounding is 2^-24 / sqrt(3) rms of the power of two below the sum; over all places between two powers of two, by their logarithm, that is
    # sqrt(0.54) of it relative to the sum.  (Parts one after the other, 29 and 31 of them, and runs by the table alone: 1.1 to 1.7 times these bounds.)
    import torch
    N = 20_000
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.arange(M, device="cuda", dtype=torch.int32).repeat_interleave(n)
    cols = torch.randint(0, N, (M, n), generator=g, device="cuda").sort(dim=1).values
    H, vals = torch.rand((N, K), generator=g, device="cuda"), torch.rand((M, n), generator=g, device="cuda")
    plan = engine.plan_coo(M, N, rows, cols.flatten().to(torch.int32), K)
    Y = torch.full((M, K), float("nan"), device="cuda")
    if fused:
        W = torch.zeros((M, K), device="cuda")
        H[:, 0], W[:, 0] = 1, 1
        plan.fused(W, H, Y, vals.flatten())
    else:
        plan.spmm(H, Y, vals.flatten())
    plan.close()
    square = 0.0
    for a in range(0, M, 200):
        ref = torch.einsum("mn,mnk->mk", vals[a:a + 200].double(), H[cols[a:a + 200]].double())
        square += float(((Y[a:a + 200].double() - ref) / ref).square().sum())
    p = n / (chain * block)
    parts = p / 3 if p <= 8 else 64 / (3 * p) + p / 24
    assert square / (M * K) <= 2.0 ** -48 / 3 * 0.54 * (chain / (3 * p) + parts + 2)


@pytest.mark.parametrize("K,N", [(388, 590_000), (416, 545_000), (644, 354_000), (900, 420_000)])
def test_long_rows_whole(engine, K, N):
    # rows that are no multiple of 128 bytes, or whose last pass would be narrow: one launch, however large H is
    import torch
    M, nnz = 7_013, 1_000_003
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    H, vals = (torch.randint(-2, 3, n, generator=g, device="cuda").float() for n in ((N, K), (nnz,)))   # every product and sum exact
    plan = engine.plan_coo(M, N, rows, cols, K)
    Y, n0 = torch.full((M, K), float("nan"), device="cuda"), engine.kernel_launches()
    plan.spmm(H, Y, vals)
    assert engine.kernel_launches() - n0 == 1
    plan.close()
    ref = torch.zeros((M, K), device="cuda")
    for a in range(0, nnz, 100_000):
        i = slice(a, a + 100_000)
        ref.index_add_(0, rows[i].long(), vals[i, None] * H[cols[i].long()])
    assert torch.equal(Y, ref)
