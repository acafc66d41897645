"""Plans used from several streams and under stream capture.

What a plan builds when a call first needs it (row pointer, scratch of SpMM, hub marks, work items) has to be complete for the
calls that follow on other streams, and may be built while a stream is captured.  Results are compared bit for bit with
the same calls made one after the other."""
import numpy as np
import pytest
import torch

from helpers import assert_parity, random_coo
from sddmm_gpu_b200 import api

pytestmark = pytest.mark.gpu


def _problem(M, N, nnz, K, seed=0):
    rng = np.random.default_rng(seed)
    rows, cols = random_coo(rng, M, N, nnz, empty_rows=[0, 7, M - 1], hub_row=5)
    vals = rng.standard_normal(rows.shape[0]).astype(np.float32)
    W, H = (rng.standard_normal((n, K)).astype(np.float32) for n in (M, N))
    return [torch.from_numpy(a).cuda() for a in (rows, cols, vals, W, H)]


def _keep_busy():
    """Work on the current stream that takes some tens of milliseconds."""
    a = torch.randn(8192, 8192, device="cuda")
    for _ in range(40):
        a = a @ a * 1e-4
    return a


@pytest.mark.parametrize("fused", [False, True])
def test_first_spmm_on_a_busy_stream_second_on_another(engine, fused):
    M, N, K = 4000, 3000, 64
    rows, cols, vals, W, H = _problem(M, N, 200_000, K)

    def call(plan, Y, flags=0):
        plan.fused(W, H, Y, vals, None, flags) if fused else plan.spmm(H, Y, vals, flags)

    reference = torch.full((M, K), float("nan"), device="cuda")
    plan = engine.plan_coo(M, N, rows, cols, K)
    call(plan, reference)
    plan.close()
    A, B = torch.cuda.Stream(), torch.cuda.Stream()
    Y = [torch.full((M, K), float("nan"), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    plan = engine.plan_coo(M, N, rows, cols, K)
    with torch.cuda.stream(A):
        busy = _keep_busy()
        call(plan, Y[0], api.FLAG_ASYNC)
    with torch.cuda.stream(B):
        assert plan.export_row_ptr()[-1] == rows.shape[0]
    with torch.cuda.stream(B):
        call(plan, Y[1], api.FLAG_ASYNC)
    torch.cuda.synchronize()
    assert torch.equal(Y[0], reference) and torch.equal(Y[1], reference)
    plan.close()
    del busy


@pytest.mark.parametrize("what", ["ring", "panel", "gather", "default", "bf16_ring", "spmm", "fused"])
def test_first_call_of_a_plan_may_be_captured(engine, what, monkeypatch):
    monkeypatch.setenv("SDDMM_L2_HUB_MB", "1")     # the ring kernel's hub marks are wanted at this size
    M, N, K = 3000, 2500, 256
    rows, cols, vals, W, H = _problem(M, N, 150_000, K)
    Wb, Hb = W.to(torch.bfloat16), H.to(torch.bfloat16)
    flags = {"ring": api.FLAG_KERNEL_RING, "panel": api.FLAG_KERNEL_PANEL, "gather": api.FLAG_KERNEL_GATHER, "default": 0,
             "bf16_ring": api.FLAG_KERNEL_RING | api.FLAG_OPERANDS_BF16}

    def call(plan, out, extra=0):
        if what == "spmm":
            plan.spmm(H, out, vals, extra)
        elif what == "fused":
            plan.fused(W, H, out, vals, None, extra)
        else:
            plan.execute(*((Wb, Hb) if what == "bf16_ring" else (W, H)), out, vals, flags[what] | extra)

    shape = (M, K) if what in ("spmm", "fused") else (rows.shape[0],)
    expect, out = (torch.full(shape, float("nan"), device="cuda") for _ in range(2))
    plan = engine.plan_coo(M, N, rows, cols, K)
    call(plan, expect)
    plan.close()
    plan = engine.plan_coo(M, N, rows, cols, K)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(plan, out, api.FLAG_ASYNC)
    assert bool(torch.isnan(out).all())            # captured, not run
    for _ in range(3):
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, expect)
    del graph
    plan.close()


def test_overlapping_spmm_calls_of_one_plan(engine):
    """Asynchronous calls alternating over three streams, rows of many partial sums: the scratch and its counters are the
    plan's, so the calls run one after the other; and the calls after them find the counters at zero."""
    M, N, K = 3000, 2500, 128
    rows, cols, vals, W, H = _problem(M, N, 400_000, K, seed=3)
    plan = engine.plan_coo(M, N, rows, cols, K)
    expect = [torch.full((M, K), float("nan"), device="cuda") for _ in range(2)]
    plan.spmm(H, expect[0], vals)
    plan.fused(W, H, expect[1], vals)
    streams = [torch.cuda.Stream() for _ in range(3)]
    out = [torch.full((M, K), float("nan"), device="cuda") for _ in range(24)]
    torch.cuda.synchronize()
    for i, Y in enumerate(out):
        with torch.cuda.stream(streams[i % 3]):
            plan.fused(W, H, Y, vals, None, api.FLAG_ASYNC) if i % 2 else plan.spmm(H, Y, vals, api.FLAG_ASYNC)
    late = torch.full((M, K), float("nan"), device="cuda")
    plan.spmm(H, late, vals)                       # waits, behind all of them
    assert torch.equal(late, expect[0])
    torch.cuda.synchronize()
    for i, Y in enumerate(out):
        assert torch.equal(Y, expect[i % 2]), i
    # a captured call between them, and its replays in order with the others
    graph, Y = torch.cuda.CUDAGraph(), torch.full((M, K), float("nan"), device="cuda")
    with torch.cuda.graph(graph):
        plan.spmm(H, Y, vals, api.FLAG_ASYNC)
    for i in range(4):
        Y.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(Y, expect[0])
        with torch.cuda.stream(streams[i % 3]):
            plan.fused(W, H, out[i], vals, None, api.FLAG_ASYNC)
        torch.cuda.synchronize()
        assert torch.equal(out[i], expect[1])
    with pytest.raises(api.SddmmError) as e:       # host arrays need the call to wait
        plan.spmm(np.zeros((N, K), np.float32), late, vals, api.FLAG_ASYNC)
    assert e.value.status == api.INVALID_ARG
    plan.close()


def test_overlapping_ring_calls(engine):
    """Asynchronous calls on two streams through the kernel whose warps take their share of the work from a counter: a large one
    is under way when a small one begins."""
    K, N = 256, 60_000
    g = torch.Generator(device="cuda").manual_seed(0)
    plans, calls = [], []
    for M, nnz in ((50_000, 12_000_000), (3_000, 40_000)):
        rows = torch.sort(torch.randint(0, M, (nnz,), generator=g, device="cuda")).values.to(torch.int32)
        cols = torch.randint(0, N, (nnz,), generator=g, device="cuda", dtype=torch.int32)
        W, H = (torch.randn((n, K), generator=g, device="cuda") for n in (M, N))
        plan, expect = engine.plan_coo(M, N, rows, cols, K), torch.empty(nnz, device="cuda")
        plan.execute(W, H, expect, None, api.FLAG_KERNEL_RING)
        plans.append((plan, rows, cols))
        calls.append((plan, W, H, expect))
    streams = [torch.cuda.Stream() for _ in calls]
    for _ in range(3):
        out = [torch.full_like(expect, float("nan")) for _, _, _, expect in calls]
        torch.cuda.synchronize()
        for stream, (plan, W, H, _), P in zip(streams, calls, out):
            with torch.cuda.stream(stream):
                plan.execute(W, H, P, None, api.FLAG_ASYNC | api.FLAG_KERNEL_RING)
        torch.cuda.synchronize()
        for P, (_, _, _, expect) in zip(out, calls):
            assert torch.equal(P, expect)
    for plan, _, _ in plans:
        plan.close()


def test_plan_destroyed_behind_a_queued_row_upload(engine):
    """The list of used rows belongs to the plan and is read by uploads on any stream: destroying the plan waits for them, and
    the memory of the list goes to the next plan only then."""
    M, N, K = 60000, 500, 32
    rng = np.random.default_rng(2)
    rows = np.sort(rng.choice(np.arange(0, M, 2), 40_000)).astype(np.int32)      # odd rows stay empty
    cols = rng.integers(0, N, rows.size).astype(np.int32)
    rows_d, cols_d = torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda()
    host = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).pin_memory()
    dev = torch.zeros((M, K), device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    plan = engine.plan_coo(M, N, rows_d, cols_d, K)
    ids, n = plan.used_lines(0)
    with torch.cuda.stream(side):
        busy = _keep_busy()
    engine.upload_rows(host, dev, ids, n, K, side.cuda_stream)
    plan.close()
    assert side.query()                            # the upload is done, the list was free to go
    others = []
    for _ in range(4):                             # plans that take memory of that size and write to it
        q = engine.plan_coo(M, N, rows_d, cols_d, K)
        q.used_lines(0)
        others.append(q)
    torch.cuda.synchronize()
    expect = np.zeros((M, K), np.float32)
    expect[rows] = host.numpy()[rows]
    assert np.array_equal(dev.cpu().numpy(), expect)
    for q in others:
        q.close()
    del busy


def test_plans_destroyed_by_another_thread(engine):
    """A garbage collector may destroy plans from any thread while the handle works: what they give back (memory, kernel clocks,
    event pairs) is shared."""
    import threading
    M, N, K = 2000, 1500, 64
    rows, cols, vals, W, H = _problem(M, N, 60_000, K)
    expect = torch.full((rows.shape[0],), float("nan"), device="cuda")
    Y = torch.full((M, K), float("nan"), device="cuda")
    plans = []
    for i in range(60):
        p = engine.plan_coo(M, N, rows, cols, K)
        p.execute(W, H, expect, vals)                                     # holds a clock
        if i % 2:
            p.execute(W, H, expect, vals, api.FLAG_KERNEL_PANEL)          # holds an event pair
        p.spmm(H, Y, vals)
        plans.append(p)
    keep = engine.plan_coo(M, N, rows, cols, K)
    keep.execute(W, H, expect, vals)
    worker = threading.Thread(target=lambda: [p.close() for p in plans])
    worker.start()
    for _ in range(200):
        out = torch.full((rows.shape[0],), float("nan"), device="cuda")
        engine.sddmm_coo(M, N, rows, cols, W, H, K, out, vals)
        assert torch.equal(out, expect)
        again = engine.plan_coo(M, N, rows, cols, K)
        again.execute(W, H, out, vals)
        assert torch.equal(out, expect) and 0 < again.last_kernel_ms() < 10
        again.close()
        if not worker.is_alive():
            break
    worker.join()
    keep.execute(W, H, out, vals)
    assert torch.equal(out, expect)
    keep.close()


def test_trim_gives_the_kept_memory_back():
    h = api.Handle(0)
    M, N, K = 40_000, 30_000, 256
    rows, cols, vals, W, H = _problem(M, N, 300_000, K)
    out = torch.zeros(rows.shape[0], device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    Wh, Hh = W.cpu(), H.cpu()
    for _ in range(3):
        h.sddmm_coo(M, N, rows, cols, Wh, Hh, K, out, vals)        # 72 MB of operands staged
    assert before - torch.cuda.mem_get_info()[0] >= 60 << 20
    h.trim()
    assert before - torch.cuda.mem_get_info()[0] < 20 << 20
    expect = out.clone()
    h.sddmm_coo(M, N, rows, cols, W, H, K, out, vals)
    assert torch.equal(out, expect)
    h.close()
