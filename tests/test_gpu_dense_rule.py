"""When a locally dense matrix goes through the dense-cell kernel (from nnz * K = 2^26 on), and that kernel at small sizes.

Tolerance: tests/helpers.py (1e-4 of max(|ref|, sum of magnitudes) per nonzero, against the CPU oracle)."""
import numpy as np
import pytest

from helpers import assert_parity
from sddmm_gpu_b200 import api, synth

pytestmark = pytest.mark.gpu


def _run(h, p, rows, cols, vals):
    plan = h.plan_coo(p["M"], p["N"], rows, cols, p["W"].shape[1])
    P = np.full(rows.shape[0], np.nan, np.float32)
    plan.execute(p["W"], p["H"], P, vals)
    name, info = plan.last_kernel_name(), plan.info()
    again = np.full(rows.shape[0], np.nan, np.float32)
    plan.execute(p["W"], p["H"], again, vals)
    assert plan.last_kernel_name() == name and np.array_equal(P, again)
    plan.close()
    assert_parity(P, rows, cols, p["W"], p["H"], vals)
    return name, info


@pytest.mark.parametrize("K", [256, 512])
def test_line_between_the_kernels(engine, K):
    p = synth.to_numpy(synth.attention_mask(M=1100, half_width=96, n_global=7, K=K, device="cpu"))
    rows, cols = p["rows"], p["cols"]
    work = rows.shape[0] * K
    name, info = _run(engine, p, rows, cols, None)
    assert (work >= 1 << 26) == (K == 512)
    assert name.startswith("dense") == (K == 512)
    # what is reported is what runs
    assert (info.n_dense_cells > 0) == (K == 512) and (info.n_dense_nnz > 0) == (K == 512) and info.n_dense_nnz <= info.nnz


@pytest.mark.parametrize("M,half_width,n_global", [(300, 64, 0), (1100, 96, 7), (4096, 96, 20)])
@pytest.mark.parametrize("mode", ["2", "1", "0"])
@pytest.mark.parametrize("K", [16, 36, 64, 100, 256])
def test_dense_cells_at_small_sizes(monkeypatch, K, mode, M, half_width, n_global):
    # a CTA with one cell, with none, with several; chunks of K that are full, ragged, single
    monkeypatch.setenv("SDDMM_DENSE_CELLS", "1")
    monkeypatch.setenv("SDDMM_DENSE_TENSOR", mode)
    h = api.Handle(0)
    p = synth.to_numpy(synth.attention_mask(M=M, half_width=half_width, n_global=n_global, K=K, device="cpu"))
    rng = np.random.default_rng(K)
    rows, cols = p["rows"], p["cols"]
    vals = rng.standard_normal(rows.shape[0]).astype(np.float32)
    order = np.lexsort((rng.random(rows.shape[0]), rows))    # columns in random order inside each row: per-nonzero lists
    for c, v in ((cols, vals), (cols, None), (cols[order], vals[order])):
        name, info = _run(h, p, rows, c, v)
        assert name.startswith("dense") and info.n_dense_cells > 0
    h.close()


@pytest.mark.parametrize("mode", ["2", "1", "0"])
@pytest.mark.parametrize("M,N,fill", [(128, 64, 1.0), (200, 64 * 3, 0.5), (390, 64 * 5 + 3, 0.3), (1300, 64, 0.9)])
def test_cells_with_several_nonzeros_in_one_place(monkeypatch, mode, M, N, fill):
    # one cell, an odd number of cells in a row of cells (a unit of one), units of rows that end in the cell; and rows in which some
    # columns come twice or three times: of those a cell holds one, the others are in the remainder
    monkeypatch.setenv("SDDMM_DENSE_CELLS", "1")
    monkeypatch.setenv("SDDMM_DENSE_TENSOR", mode)
    h = api.Handle(0)
    rng = np.random.default_rng(M)
    K = 72
    W, H = (rng.standard_normal((n, K)).astype(np.float32) for n in (M, N))
    cells = rng.random((M, N)) < fill
    for extra in (0, M // 2):
        rows, cols = np.nonzero(cells)
        again = rng.integers(0, rows.size, extra)
        again = np.concatenate([again, again[: extra // 3]])
        rows, cols = np.concatenate([rows, rows[again]]), np.concatenate([cols, cols[again]])
        order = np.lexsort((cols, rows))
        rows, cols = rows[order].astype(np.int32), cols[order].astype(np.int32)
        vals = rng.standard_normal(rows.size).astype(np.float32)
        name, info = _run(h, dict(M=M, N=N, W=W, H=H), rows, cols, vals)
        assert name.startswith("dense") and 0 < info.n_dense_nnz <= rows.size - again.size
    h.close()


@pytest.mark.parametrize("mode", ["2", "1", "0"])
@pytest.mark.parametrize("M,half_width,full", [(1300, 128, (300, 310)), (700, 64, (0, 5, 9, 130, 135, 140, 699)), (600, 96, (100, 101, 120, 121, 122, 180))])
def test_cells_with_columns_in_other_cells(monkeypatch, mode, M, half_width, full):
    # a band and a few full columns: the full ones are taken out of the band's cells, whose rows then have several gaps in their input positions.  Position and column
    # go up together all the same, so none of them needs a table (32 KB); the full columns, fewer than a quarter of a cell, are in the remainder
    import torch
    monkeypatch.setenv("SDDMM_DENSE_CELLS", "1")
    monkeypatch.setenv("SDDMM_DENSE_TENSOR", mode)
    h = api.Handle(0)
    K = 40
    at = torch.arange(M, device="cuda")
    cells = (at[:, None] - at).abs() <= half_width
    cells[:, list(full)] = True
    rows, cols = (a.to(torch.int32).contiguous() for a in cells.nonzero().T)
    g = torch.Generator(device="cuda").manual_seed(M)
    W, H = (torch.randint(-2, 3, (M, K), generator=g, device="cuda").float() for _ in range(2))   # every product and sum exact
    S = torch.randint(-3, 4, rows.shape, generator=g, device="cuda").float()
    plan = h.plan_coo(M, M, rows, cols, K)
    info = plan.info()
    assert info.n_dense_cells > 0 and info.nnz - info.n_dense_nnz >= len(full) * M // 2
    assert info.device_bytes < (24 + 2560 + 32) * info.n_dense_cells + 12 * (info.nnz - info.n_dense_nnz) + 8 * (M + 1) + 32768
    ref = (W @ H.T)[rows.long(), cols.long()]
    for v in (S, None):
        P = torch.full(rows.shape, float("nan"), device="cuda")
        plan.execute(W, H, P, v)
        assert plan.last_kernel_name().startswith("dense") and torch.equal(P, ref if v is None else ref * v)
    plan.close()
    h.close()


@pytest.mark.parametrize("K,half_width,n_global", [(64, 96, 6), (100, 40, 60), (512, 70, 3)])
def test_remainder_beside_the_cells(engine, K, half_width, n_global):
    # the remainder runs beside the dense cells: what follows on the stream sees all of P, and the next call overwrites it
    # only after that
    import torch
    p = synth.attention_mask(M=8192, half_width=half_width, n_global=n_global, K=K, device="cuda")
    plan = engine.plan_coo(p["M"], p["N"], p["rows"], p["cols"], K)
    info = plan.info()
    assert 0 < info.n_dense_nnz < info.nnz
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        P = torch.empty(info.nnz, device="cuda")
        seen = []
        for _ in range(6):
            P.fill_(float("nan"))
            plan.execute(p["W"], p["H"], P, p["vals"], api.FLAG_ASYNC)
            seen.append(P.clone())
    stream.synchronize()
    assert plan.last_kernel_name() == "dense_tc+gather"
    q = synth.to_numpy(p)
    assert_parity(seen[0].cpu().numpy(), q["rows"], q["cols"], q["W"], q["H"], q["vals"])
    assert all(torch.equal(seen[0], s) for s in seen[1:])
    plan.close()


@pytest.mark.parametrize("where", ["pageable", "pinned", "device"])
def test_unsorted_rows_behind_skipped_validation(engine, where, monkeypatch):
    # blocks of full rows in descending order, long rows and enough work for dense cells: only sddmm_execute, which looks at a
    # nonzero at a time, takes them, and goes by no row pointer
    import torch
    monkeypatch.setenv("SDDMM_DENSE_CELLS", "1")
    M, N, K = 700, 300, 64
    rng = np.random.default_rng(4)
    rows = np.repeat(np.arange(M - 1, -1, -1), 200).astype(np.int32)
    cols = np.concatenate([np.sort(rng.choice(N, 200, replace=False)) for _ in range(M)]).astype(np.int32)
    vals = rng.standard_normal(rows.size).astype(np.float32)
    W, H = (rng.standard_normal((n, K)).astype(np.float32) for n in (M, N))
    plan = engine.plan_coo(M, N, rows, cols, K, flags=api.PLAN_SKIP_VALIDATION)
    P = np.full(rows.size, np.nan, np.float32)
    args = [torch.from_numpy(a) for a in (W, H, P, vals)]
    if where == "pinned":
        args = [a.pin_memory() for a in args]
    elif where == "device":
        args = [a.cuda() for a in args]
    plan.execute(*args)
    assert_parity(args[2].cpu().numpy(), rows, cols, W, H, vals)
    Y = np.zeros((M, K), np.float32)
    for refused in (lambda: plan.spmm(H, Y, vals), lambda: plan.fused(W, H, Y, vals), lambda: plan.used_lines(0), plan.export_row_ptr):
        with pytest.raises(api.SddmmError) as e:
            refused()
        assert e.value.status == api.UNSORTED_INPUT
    assert plan.used_lines(1)[1] == np.unique(cols).size
    plan.close()
