"""The gather kernel (csrc/sddmm_gather.cu) at the edges of its lane shapes, and the timing of small calls.

Tolerance: tests/helpers.py (1e-4 of max(|ref|, sum of magnitudes) per nonzero, against the CPU oracle)."""
import numpy as np
import pytest
import torch

from helpers import assert_parity, random_coo
from sddmm_gpu_b200 import api

pytestmark = pytest.mark.gpu

# the first and last K of every lane shape, exact widths, and the long-row form (K > 1024)
EDGES = [4, 16, 20, 28, 32, 36, 48, 52, 60, 64, 68, 96, 100, 124, 128, 132, 192, 196, 252, 256, 260, 320, 324, 384, 388, 508,
         512, 516, 640, 644, 768, 772, 896, 900, 1024, 1028, 1536, 4096]


@pytest.mark.parametrize("K", EDGES)
def test_gather_shapes(engine, K):
    rng = np.random.default_rng(K)
    M, N = 97, 131
    # one nonzero; less than a step; a partial step behind full ones; one row; rows that change at every nonzero
    for nnz, hub in ((1, None), (7, None), (1031, None), (2000, 40)):
        rows, cols = random_coo(rng, M, N, nnz, empty_rows=[0, 3, M - 1], hub_row=hub)
        if rows.size == 0:
            continue
        vals = rng.standard_normal(rows.shape[0]).astype(np.float32)
        W = rng.standard_normal((M, K)).astype(np.float32)
        H = rng.standard_normal((N, K)).astype(np.float32)
        for col_tile in (0, 50):   # 50: the nonzeros in tiled order, results through the permutation
            plan = engine.plan_coo(M, N, rows, cols, K, 0, col_tile)
            for sv in (vals, None):
                P = np.full(rows.shape[0], np.nan, np.float32)
                plan.execute(W, H, P, sv)
                assert_parity(P, rows, cols, W, H, sv)
            plan.close()
        P = np.full(rows.shape[0], np.nan, np.float32)
        engine.sddmm_coo(M, N, rows, cols, W, H, K, P, vals)
        assert_parity(P, rows, cols, W, H, vals)


@pytest.mark.parametrize("K", [4, 16, 28, 32, 44, 48, 60, 64, 96, 100, 128, 160, 192, 200, 256, 300, 380, 384, 500, 512])
def test_few_nonzeros_as_many(engine, K):
    # calls of at most 10 MB of H rows that are waited for have a kernel of their own: the same bits as the same nonzeros at the front of a call that is larger
    M, N = 900, 1100
    most = 10_000_000 // (4 * K)
    g = torch.Generator(device="cuda").manual_seed(K)
    nnz = most + 5000
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    W, H, S = (torch.randn(n, generator=g, device="cuda") for n in ((M, K), (N, K), (nnz,)))
    W[M // 2, 1], H[3, 0], S[1] = float("inf"), float("nan"), float("-inf")
    many = {}
    for sv in (S, None):
        many[sv is None] = torch.full((nnz,), 7.0, device="cuda")
        plan = engine.plan_coo(M, N, rows, cols, K)
        plan.execute(W, H, many[sv is None], sv)
        plan.close()
    for n in (1, 2, 3, 9, 63, 65, 1000, most - 1, most, most + 1):
        plan = engine.plan_coo(M, N, rows[:n], cols[:n], K)
        for sv in (S, None):
            P = torch.full((n + 1,), 7.0, device="cuda")
            plan.execute(W, H, P[:n], None if sv is None else sv[:n])
            assert torch.equal(P[:n].view(torch.int32), many[sv is None][:n].view(torch.int32)) and float(P[n]) == 7.0
            assert plan.last_kernel_ms() > 0
            engine.sddmm_coo(M, N, rows[:n], cols[:n], W, H, K, P[:n], None if sv is None else sv[:n])
            assert torch.equal(P[:n].view(torch.int32), many[sv is None][:n].view(torch.int32)) and float(P[n]) == 7.0
        plan.close()


@pytest.mark.parametrize("K", [52, 60, 64, 512])
def test_few_waves_as_many(engine, K):
    # 52 to 64 columns: from 208,384 to 303,103 nonzeros of 148 SMs and from 397,824 to 454,655 take four rows at a time, K = 512: from 37,888 to 56,831 and from 75,776
    # to 85,247 two: the same bits as the front of a call of many
    M, N, nnz = 9_001, 7_001, 600_000
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    W, H, S = (torch.randn(n, generator=g, device="cuda") for n in ((M, K), (N, K), (nnz,)))
    P = {}
    for n in (nnz, 37_887, 37_888, 50_001, 56_831, 56_832, 75_776, 85_248, 151_552, 208_383, 208_384, 213_119, 300_001, 303_103, 303_104, 397_823, 397_824, 454_655, 454_656, 473_599, 473_600):
        plan = engine.plan_coo(M, N, rows[:n], cols[:n], K)
        P[n] = torch.full((n + 1,), 7.0, device="cuda")
        plan.execute(W, H, P[n][:n], S[:n])
        plan.close()
        assert torch.equal(P[n][:n], P[nnz][:n]) and float(P[n][n]) == 7.0


@pytest.mark.parametrize("K,N", [(100, 20_000), (124, 16_130), (124, 16_128), (64, 20_000), (60, 20_000)])
def test_many_nonzeros_of_a_large_h(engine, K, N):
    # from a million nonzeros and 8 MB of H on rows of 100 to 124 columns have a shape of their own (16,128 rows are below); the chunks of a call with host
    # operands are summed as the whole.  Small whole numbers: every product and sum is exact.
    M, nnz = 200_003, 1_000_003
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    W, H, S = (torch.randint(-2, 3, n, generator=g, device="cuda").float() for n in ((M, K), (N, K), (nnz,)))
    ref = torch.cat([torch.einsum("nk,nk->n", W[rows[i:i + 100_000].long()], H[cols[i:i + 100_000].long()]) for i in range(0, nnz, 100_000)])
    plan = engine.plan_coo(M, N, rows, cols, K)
    tiled = engine.plan_coo(M, N, rows, cols, K, 0, N // 3)
    for p, sv, flags in ((plan, S, 0), (plan, None, 0), (plan, S, api.FLAG_KERNEL_GATHER), (tiled, S, 0)):
        P = torch.full((nnz,), float("nan"), device="cuda")
        p.execute(W, H, P, sv, flags)
        assert torch.equal(P, ref if sv is None else ref * sv)
    P = torch.full((nnz,), float("nan"), device="cuda")
    engine.sddmm_coo(M, N, rows, cols, W, H, K, P, S)
    assert torch.equal(P, ref * S)
    W, H = torch.randn((M, K), generator=g, device="cuda"), torch.randn((N, K), generator=g, device="cuda")
    plan.execute(W, H, P, S)
    on_host = [a.cpu().pin_memory() for a in (W, H, S, torch.zeros(nnz))]
    plan.execute(on_host[0], on_host[1], on_host[3], on_host[2])
    assert torch.equal(P.cpu(), on_host[3])
    forced = torch.full((nnz,), float("nan"), device="cuda")
    plan.execute(W, H, forced, S, api.FLAG_KERNEL_GATHER)   # the same shape
    assert torch.equal(P, forced)
    plan.close()
    tiled.close()


@pytest.mark.parametrize("K,N", [(52, 2_403_847), (60, 2_083_334), (64, 1_953_125), (64, 1_953_124)])
def test_rows_of_a_very_large_h(engine, K, N):
    # 52 to 64 columns of an H of 500 MB and more (the last N is below) have the shape of the passes; whole numbers: every product and sum is exact
    M, nnz = 50_021, 600_011
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    cols[-1] = N - 1
    W, H, S = (torch.randint(-2, 3, n, generator=g, device="cuda").float() for n in ((M, K), (N, K), (nnz,)))
    ref = torch.cat([torch.einsum("nk,nk->n", W[rows[i:i + 100_000].long()], H[cols[i:i + 100_000].long()]) for i in range(0, nnz, 100_000)]) * S
    plan = engine.plan_coo(M, N, rows, cols, K)
    for flags in (0, api.FLAG_KERNEL_GATHER):
        P = torch.full((nnz + 1,), 7.0, device="cuda")
        plan.execute(W, H, P[:nnz], S, flags)
        assert torch.equal(P[:nnz], ref) and float(P[nnz]) == 7.0
    plan.close()


def test_kernel_time_of_small_calls(engine):
    # timed by the kernel's own clock; each plan keeps its own time, also when calls of other plans lie between, and an
    # asynchronous call has none
    rng = np.random.default_rng(1)
    plans = []
    for nnz in (500, 60000):
        rows, cols = random_coo(rng, 400, 300, nnz)
        t = [torch.from_numpy(a).cuda() for a in (rows, cols)]
        ops = [torch.randn(n, 64, device="cuda") for n in (400, 300)]
        plans.append((engine.plan_coo(400, 300, *t, 64), ops, torch.zeros(rows.shape[0], device="cuda")))
    for _ in range(3):
        for plan, (W, H), P in plans:
            plan.execute(W, H, P)
    times = [plan.last_kernel_ms() for plan, _, _ in plans]
    assert all(0 < t < 1.0 for t in times)
    assert times == [plan.last_kernel_ms() for plan, _, _ in plans]
    plan, (W, H), P = plans[0]
    plan.execute(W, H, P, None, api.FLAG_ASYNC)
    assert plan.last_kernel_ms() == -1.0
    assert plans[1][0].last_kernel_ms() == times[1]
    for plan, _, _ in plans:
        plan.close()


def _all_of_P(engine, M, N, nnz, K):
    """A call of nnz nonzeros with small whole-number operands (every product and sum exact): P against W H^T, everywhere.
    Returns the plan's kernel time and the whole call's, in ms."""
    g = torch.Generator(device="cuda").manual_seed(nnz % 1009)
    j = torch.arange(nnz, device="cuda")
    rows, cols = (j * M // nnz).to(torch.int32), (j % N).to(torch.int32)
    del j
    W, H = (torch.randint(-2, 3, (n, K), generator=g, device="cuda").float() for n in (M, N))
    plan = engine.plan_coo(M, N, rows, cols, K)
    P = torch.full((nnz,), float("nan"), device="cuda")
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t0.record()
    plan.execute(W, H, P)
    t1.record()
    torch.cuda.synchronize()
    ms = plan.last_kernel_ms()
    plan.close()
    table = (W.double() @ H.double().T).float()
    for a in range(0, nnz, 1 << 27):
        b = min(nnz, a + (1 << 27))
        assert torch.equal(P[a:b], table[rows[a:b].long(), cols[a:b].long()]), (a, b)
    return ms, t0.elapsed_time(t1)


def test_long_rows_beyond_two_to_the_27_nonzeros(engine, monkeypatch):
    # K > 1024: a warp per nonzero, 2^32 threads at 2^27 nonzeros
    monkeypatch.setenv("SDDMM_DENSE_CELLS", "0")   # every cell of these few rows and columns is full
    _all_of_P(engine, 512, 509, (1 << 27) + 12345, 1028)


def test_kernel_time_covers_all_launches(engine, monkeypatch):
    # more than 2^30 nonzeros go out in two launches
    monkeypatch.setenv("SDDMM_DENSE_CELLS", "0")
    ms, around = _all_of_P(engine, 512, 509, (1 << 30) + 54321, 4)
    assert 0.9 * around <= ms <= around


@pytest.mark.parametrize("K,N,bf16", [(324, 310_000, False), (416, 2_100_000, False), (512, 489_000, False), (772, 131_000, False),
                                      (1028, 98_000, False), (1024, 930_000, True)])
def test_long_rows_in_passes(engine, K, N, bf16):
    # large H, long rows: passes over part of the columns, the later ones adding to P.  The last pass narrower than the others, rows of
    # one and of many nonzeros, a nonzero count that ends inside a step; against fp64 on the GPU and against the call in one pass
    M, nnz = 20_011, 1_000_003
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda") ** 2 // M).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    W, H = (torch.randn((n, K), generator=g, device="cuda") for n in (M, N))
    vals = torch.randn(nnz, generator=g, device="cuda")
    flag = 0
    if bf16:
        W, H, flag = W.bfloat16(), H.bfloat16(), api.FLAG_OPERANDS_BF16
    plan = engine.plan_coo(M, N, rows, cols, K)
    ref, mag = torch.empty(nnz, device="cuda", dtype=torch.float64), torch.empty(nnz, device="cuda", dtype=torch.float64)
    for a in range(0, nnz, 50_000):
        i = slice(a, min(nnz, a + 50_000))
        t = W[rows[i].long()].double() * H[cols[i].long()].double()
        ref[i], mag[i] = t.sum(1), t.abs().sum(1)
    n0 = engine.kernel_launches()
    for S in (None, vals):
        P = torch.full((nnz,), float("nan"), device="cuda")
        plan.execute(W, H, P, S, flag)
        s = 1.0 if S is None else S.double()
        # K products and sums in fp32, and one more rounding for S
        assert bool(((P.double() - ref * s).abs() <= (K + 2) * 2.0 ** -24 * (mag * s).abs()).all())
        assert plan.last_kernel_ms() > 0
    assert engine.kernel_launches() - n0 >= 4      # passes, not one launch each
    # S and P in one array: the S values have to outlive the first pass
    both = vals.clone()
    plan.execute(W, H, both, both, flag)
    assert bool(((both.double() - ref * vals.double()).abs() <= (K + 2) * 2.0 ** -24 * (mag * vals.double()).abs()).all())
    # not finite: in one row of H, and in one S value
    c = int(cols[5])
    H[c, K - 1] = float("inf")
    vals[9] = float("nan")
    plan.execute(W, H, P, vals, flag)
    want = torch.isfinite(vals) & (cols != c)
    assert torch.equal(torch.isfinite(P), want)
    if not bf16:
        whole = torch.empty_like(P)
        plan.execute(W, H, whole, vals, api.FLAG_KERNEL_GATHER)
        assert torch.equal(torch.isfinite(whole), want)
    plan.close()


def test_tiled_order_in_passes(engine):
    # a column-tiled plan asked for its own order has no permutation: passes as in input order, timed as a whole
    K, M, N, nnz, tile = 768, 60_013, 150_011, 4_000_003, 70_000
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    W, H = (torch.randint(-2, 3, (n, K), generator=g, device="cuda").float() for n in (M, N))   # every product and sum exact
    plan = engine.plan_coo(M, N, rows, cols, K, 0, tile)
    P = torch.full((nnz,), float("nan"), device="cuda")
    for _ in range(2):
        n0 = engine.kernel_launches()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        plan.execute(W, H, P, None, api.FLAG_TILED_ORDER)
        t1.record()
        torch.cuda.synchronize()
        assert engine.kernel_launches() - n0 == 4
    # the four passes take milliseconds, of which a launch and a wait are tens of microseconds
    assert 0.9 * t0.elapsed_time(t1) <= plan.last_kernel_ms() <= t0.elapsed_time(t1)
    order = torch.argsort(cols // tile, stable=True)
    for a in range(0, nnz, 200_000):
        i = order[a:a + 200_000]
        assert torch.equal(P[a:a + 200_000], (W[rows[i].long()] * H[cols[i].long()]).sum(1)), a
    plan.close()


@pytest.mark.parametrize("K,N,bf16", [(768, 131_000, False), (1024, 930_000, True)])
def test_subnormal_sums_in_passes(engine, K, N, bf16):
    # products that are multiples of 2^-142 and whose sums stay below 2^-126: exact in fp32 as long as no pass makes zeros of them
    M, nnz = 20_011, 1_000_003
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    W, H = (torch.randint(-2, 3, (n, K), generator=g, device="cuda").float() * 2.0 ** -71 for n in (M, N))
    flag = 0
    if bf16:
        W, H, flag = W.bfloat16(), H.bfloat16(), api.FLAG_OPERANDS_BF16
    plan = engine.plan_coo(M, N, rows, cols, K)
    S = torch.full((nnz,), 2.0 ** 100, device="cuda")
    n0 = engine.kernel_launches()
    P, scaled = (torch.full((nnz,), float("nan"), device="cuda") for _ in range(2))
    plan.execute(W, H, P, None, flag)
    plan.execute(W, H, scaled, S, flag)
    assert engine.kernel_launches() - n0 == 2 * 4      # three later passes, two of them between the first and the last
    for a in range(0, nnz, 200_000):
        i = slice(a, a + 200_000)
        ref = (W[rows[i].long()].double() * H[cols[i].long()].double()).sum(1)
        assert torch.equal(P[i].double(), ref) and torch.equal(scaled[i].double(), ref * 2.0 ** 100)
    plan.close()


def _sampled_pattern(M, N, nnz, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
    return rows, torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)


@pytest.mark.parametrize("K,N,edges", [(512, 790_000, (131_071, 131_073, 999_999)), (1024, 394_000, (65_535, 65_539, 999_999))])
def test_few_nonzeros_of_a_large_H(engine, K, N, edges):
    # rows of 2 KB and more of an H of 1.6 GB: from 256 MB of rows to a million nonzeros the ring kernel, on whole rows, as the gather kernel below
    M = 20_011
    W, H = (torch.randint(-2, 3, (n, K), device="cuda").float() for n in (M, N))   # every product and sum exact
    for nnz, kernel in zip(edges, ("gather", "ring", "ring")):
        rows, cols = _sampled_pattern(M, N, nnz, nnz)
        S = torch.randint(-3, 4, (nnz,), device="cuda").float()
        plan = engine.plan_coo(M, N, rows, cols, K)
        n0 = engine.kernel_launches()
        P, inside = torch.full((nnz,), float("nan"), device="cuda"), S.clone()
        plan.execute(W, H, P, S)
        assert plan.last_kernel_name() == kernel and engine.kernel_launches() - n0 == 1 and plan.last_kernel_ms() > 0
        plan.execute(W, H, inside, inside)     # S and P in one array
        for a in range(0, nnz, 100_000):
            i = slice(a, a + 100_000)
            assert torch.equal(P[i], (W[rows[i].long()] * H[cols[i].long()]).sum(1) * S[i]), a
        assert torch.equal(P, inside)
        plan.close()


def test_few_nonzeros_of_a_large_bf16_H(engine):
    # whole rows through the gather kernel and through the ring kernel, one launch each; four passes from a million nonzeros on
    M, N, K = 20_011, 930_000, 1024
    W, H = (torch.randint(-2, 3, (n, K), device="cuda").bfloat16() for n in (M, N))   # every product and sum exact
    for nnz, kernel, launches in ((20_001, "gather", 1), (131_073, "ring", 1), (999_999, "ring", 1), (1_000_001, "gather", 4)):
        rows, cols = _sampled_pattern(M, N, nnz, nnz)
        plan = engine.plan_coo(M, N, rows, cols, K)
        P, n0 = torch.full((nnz,), float("nan"), device="cuda"), engine.kernel_launches()
        plan.execute(W, H, P, None, api.FLAG_OPERANDS_BF16)
        assert plan.last_kernel_name() == kernel + " (bf16 operands)" and engine.kernel_launches() - n0 == launches
        for a in range(0, nnz, 100_000):
            i = slice(a, a + 100_000)
            assert torch.equal(P[i], (W[rows[i].long()].float() * H[cols[i].long()].float()).sum(1)), a
        plan.close()


@pytest.mark.parametrize("K,N,nnz,passes", [(388, 260_000, 1_000_003, 1), (580, 440_000, 1_000_003, 1), (780, 330_000, 1_000_003, 1), (260, 3_850_000, 61_600_003, 1),
                                            (320, 3_126_000, 50_016_003, 5), (900, 280_000, 1_000_003, 5), (576, 440_000, 1_000_003, 3)])
def test_passes_by_the_lines_of_a_row(engine, K, N, nnz, passes):
    # rows that are no multiple of 128 bytes are multiplied whole, but for the widths at which passes pay all the same
    M = 20_011
    W, H = (torch.randint(-2, 3, (n, K), device="cuda").float() for n in (M, N))   # every product and sum exact
    rows, cols = _sampled_pattern(M, N, nnz, K)
    plan = engine.plan_coo(M, N, rows, cols, K)
    P, n0 = torch.full((nnz,), float("nan"), device="cuda"), engine.kernel_launches()
    plan.execute(W, H, P)
    assert plan.last_kernel_name() == "gather" and engine.kernel_launches() - n0 == passes and plan.last_kernel_ms() > 0
    step = -(-nnz // 1_000_003)        # of the largest every 50th and every 62nd
    for a in range(0, nnz, 100_000 * step):
        i = slice(a, a + 100_000 * step, step)
        assert torch.equal(P[i], (W[rows[i].long()] * H[cols[i].long()]).sum(1)), a
    assert not torch.isnan(P).any()
    plan.close()


def test_tiled_order_of_a_large_H(engine):
    # K = 256 and an H that input order multiplies in four passes: whole rows in the order of column tiles
    K, M, N = 256, 20_011, 3_910_001
    nnz = 16 * N + 5
    rows, cols = _sampled_pattern(M, N, nnz, K)
    W, H = (torch.randint(-2, 3, (n, K), device="cuda").float() for n in (M, N))   # every product and sum exact
    plan = engine.plan_coo(M, N, rows, cols, K, 0, 1_000_000)
    order = torch.argsort(cols // 1_000_000, stable=True)
    P, n0 = torch.full((nnz,), float("nan"), device="cuda"), engine.kernel_launches()
    plan.execute(W, H, P, None, api.FLAG_TILED_ORDER)
    assert plan.last_kernel_name() == "gather" and engine.kernel_launches() - n0 == 1 and not torch.isnan(P).any()
    plan.close()
    for a in range(0, nnz, 6_300_000):
        i = order[a:a + 6_300_000:63]
        assert torch.equal(P[a:a + 6_300_000:63], (W[rows[i].long()] * H[cols[i].long()]).sum(1)), a


@pytest.mark.parametrize("K,N,width,bf16", [(768, 131_000, 192, False), (1024, 930_000, 256, True)])
def test_parts_of_all_sizes_in_passes(engine, K, N, width, bf16):
    # the parts that the passes add: zero, subnormal, either side of the line between the two ways of adding, and ordinary, in every order.  Each part is exact, so the
    # sum is off by three roundings; where all parts are subnormal by none at all (the bound is below the smallest number then)
    M, nnz, blocks = 20_011, 1_000_003, K // width
    g = torch.Generator(device="cuda").manual_seed(K)
    rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
    cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    W, H = (torch.randint(-2, 3, (n, K), generator=g, device="cuda").float() for n in (M, N))
    size = torch.tensor([0.0, 2.0 ** -70, 2.0 ** -50, 2.0 ** -40, 2.0 ** -38, 2.0 ** -30, 1.0], device="cuda")
    W = (W.view(M, blocks, width) * size[torch.randint(0, 7, (M, blocks, 1), generator=g, device="cuda")]).view(M, K)
    H *= 2.0 ** -70
    flag = 0
    if bf16:
        W, H, flag = W.bfloat16(), H.bfloat16(), api.FLAG_OPERANDS_BF16
    plan = engine.plan_coo(M, N, rows, cols, K)
    P, n0 = torch.full((nnz,), float("nan"), device="cuda"), engine.kernel_launches()
    plan.execute(W, H, P, None, flag)
    assert engine.kernel_launches() - n0 == blocks
    plan.close()
    for a in range(0, nnz, 200_000):
        i = slice(a, a + 200_000)
        parts = (W[rows[i].long()].double() * H[cols[i].long()].double()).view(-1, blocks, width).sum(2)
        assert bool(((P[i].double() - parts.sum(1)).abs() <= 4 * 2.0 ** -24 * parts.abs().sum(1)).all()), a
