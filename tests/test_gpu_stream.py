"""The stream kernel (one warp per block-row piece, warp-level MMAs) against the CPU oracle, with and without a plan, at
the sizes where its pieces, column tiles and slabs have their edges."""
import numpy as np
import pytest

import oracle
import smat_b200 as S

pytestmark = pytest.mark.gpu
TOL = 1e-2


def _blocks(rng, counts, Kb):
    brp = np.zeros(len(counts) + 1, np.int32)
    brp[1:] = np.cumsum(counts)
    bci = np.concatenate([np.sort(rng.choice(Kb, c, replace=False)) for c in counts] or [[]]).astype(np.int32) * 16
    return brp, bci, (rng.standard_normal(brp[-1] * 256) * 0.25).astype(np.float16)


def _multiply(brp, bci, bv, B_nk, M, K, plan, hint=136):
    N = B_nk.shape[0]
    A, B, C = S.SparseMatrix.from_bcsr(M, K, brp, bci, bv), S.Matrix.from_host(B_nk), S.Matrix(M, N, fill=float("nan"))
    S.set_variant(5)
    try:
        if plan:
            p = S.Plan(A, n_hint=min(N, hint))  # wider products than the hint rounded up to 128 go in several passes
            assert p.info()["kernel"] == "spmm_bcsr_stream_kernel"
            p.set_values()
            p.spmm(B, C, check=True)
            first = C.data.clone()
            p.spmm(B, C, check=True)  # counters and scratch of the first launch are ready for the next
            assert bool((first == C.data).all())
            p.close()
        else:
            S.spmm(A, B, C, check=True)
    finally:
        S.set_variant(0)
    return C.data.cpu().numpy()


def _close(C, brp, bci, bv, B_nk, M, K):
    N = B_nk.shape[0]
    ref = oracle.bcsr_spmm(bv, brp, bci, B_nk, M, N, K, threads=8).astype(np.float16).astype(np.float32)
    mag = oracle.bcsr_spmm(np.abs(bv), brp, bci, np.abs(B_nk), M, N, K, threads=8)
    return float(np.max(np.abs(C.astype(np.float32) - ref) / (np.maximum(np.abs(ref), 1e-2 * mag) + 1e-30))) <= TOL


@pytest.mark.parametrize("plan", [False, True])
@pytest.mark.parametrize("Mb,Kb,most,N", [
    (1, 1, 1, 8),           # one block
    (5, 40, 9, 24),         # fewer octets than a tile
    (300, 64, 20, 72),      # column tiles of 40 and 32
    (40, 700, 33, 136),     # 32 column indices at a time, and one more
    (64, 512, 400, 200),    # several warps per block-row, B as slabs
    (3, 3000, 2900, 64),    # long block-rows in pieces
    (700, 6000, 90, 16),    # a narrow C
])
def test_stream_kernel_matches_oracle(Mb, Kb, most, N, plan):
    rng = np.random.default_rng(Mb + Kb + N)
    counts = rng.integers(0, most + 1, Mb)
    counts[-1] = most
    if Mb > 100:
        counts[Mb // 2] = min(Kb, 40 * most)  # one block-row far longer than the rest
    brp, bci, bv = _blocks(rng, counts, Kb)
    B_nk = rng.standard_normal((N, Kb * 16)).astype(np.float16)
    C = _multiply(brp, bci, bv, B_nk, Mb * 16, Kb * 16, plan)
    assert np.all(C.reshape(Mb, -1)[counts == 0] == 0)
    assert _close(C, brp, bci, bv, B_nk, Mb * 16, Kb * 16)


def test_stream_plan_of_a_range_and_host_buffers():
    """A plan for block-rows [b0, b1) and its host-buffer product, whose last chunk goes range by range."""
    import torch
    rng = np.random.default_rng(3)
    Mb, Kb, N, b0, b1 = 400, 300, 200, 37, 391
    brp, bci, bv = _blocks(rng, rng.integers(0, 60, Mb), Kb)
    B_nk = rng.standard_normal((N, Kb * 16)).astype(np.float16)
    A = S.SparseMatrix.from_bcsr(Mb * 16, Kb * 16, brp, bci, bv)
    S.set_variant(5)
    try:
        p = S.Plan(A, b0, b1, n_hint=N)
    finally:
        S.set_variant(0)
    rows = (b1 - b0) * 16
    C = S.Matrix(rows, N, fill=float("nan"))
    p.spmm(S.Matrix.from_host(B_nk), C, check=True)
    B_host, C_host = torch.from_numpy(B_nk.view(np.int16)).pin_memory(), torch.full((rows, N), -1, dtype=torch.int16).pin_memory()
    p.spmm_host(B_host, C_host)
    torch.cuda.synchronize()
    p.close()
    ref = oracle.bcsr_spmm(bv, brp, bci, B_nk, Mb * 16, N, Kb * 16, b0, b1).astype(np.float16).astype(np.float32)
    mag = oracle.bcsr_spmm(np.abs(bv), brp, bci, np.abs(B_nk), Mb * 16, N, Kb * 16, b0, b1)
    for got in (C.data.cpu().numpy(), C_host.numpy().view(np.float16)):
        assert float(np.max(np.abs(got.astype(np.float32) - ref) / (np.maximum(np.abs(ref), 1e-2 * mag) + 1e-30))) <= TOL


@pytest.mark.parametrize("Mb,Kb,most,hint,N", [
    (64, 512, 400, 16, 328),   # three passes, the slabs of one reused by the next, long block-rows in pieces
    (40, 100, 9, 16, 264),     # no slabs; a last pass of eight columns
    (3, 3000, 2900, 136, 600),  # passes of 256 columns, every block-row in pieces
])
def test_products_in_several_passes(Mb, Kb, most, hint, N):
    rng = np.random.default_rng(N)
    counts = rng.integers(0, most + 1, Mb)
    counts[-1] = most
    brp, bci, bv = _blocks(rng, counts, Kb)
    B_nk = rng.standard_normal((N, Kb * 16)).astype(np.float16)
    assert _close(_multiply(brp, bci, bv, B_nk, Mb * 16, Kb * 16, True, hint), brp, bci, bv, B_nk, Mb * 16, Kb * 16)


def test_plan_used_at_other_widths_than_its_hint():
    """A plan made for 16 columns of a block-sparse layer multiplies wide products with the kernel a plan made for them takes
    (one or two launches, not one or two per 128 columns) and narrow ones with its own, also after a change of values,
    from host buffers, and in a captured sequence that is replayed after the values changed again."""
    import torch
    rng = np.random.default_rng(12)
    Mb, Kb = 192, 256
    brp, bci, bv = _blocks(rng, rng.binomial(Kb, 0.2, Mb), Kb)
    M, K = Mb * 16, Kb * 16
    A = S.SparseMatrix.from_bcsr(M, K, brp, bci, bv)
    plan, wide = S.Plan(A, n_hint=16), S.Plan(A, n_hint=1024)
    assert plan.info()["kernel"] == "spmm_bcsr_stream_kernel" and wide.info()["kernel"] != "spmm_bcsr_stream_kernel"
    wide.close()
    B_nk = rng.standard_normal((1024, K)).astype(np.float16)
    widths = (8, 16, 64, 136, 520, 1024)
    B = {N: S.Matrix.from_host(B_nk[:N]) for N in widths}
    C = {N: S.Matrix(M, N, fill=float("nan")) for N in widths}

    def check(N, got, values):
        assert _close(got[:, :64], brp, bci, values, B_nk[:min(N, 64)], M, K)  # every column by the same arithmetic: a sample
        if N > 64:
            assert _close(got[:, N - 64:], brp, bci, values, B_nk[N - 64:N], M, K)

    values = bv
    for scale in (1.0, -2.0):
        if scale != 1.0:
            A.bcsrVal.mul_(scale)
            plan.set_values()
            values = (values * np.float16(scale)).astype(np.float16)
        for N in widths:
            before = S.launch_count()
            plan.spmm(B[N], C[N], check=True)
            assert S.launch_count() - before <= 2
            check(N, C[N].data.cpu().numpy(), values)
    for N in (16, 1024):
        B_host, C_host = torch.from_numpy(B_nk[:N].view(np.int16)).pin_memory(), torch.full((M, N), -1, dtype=torch.int16).pin_memory()
        plan.spmm_host(B_host, C_host)
        torch.cuda.synchronize()
        check(N, C_host.numpy().view(np.float16), values)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.set_values()
        for N in (16, 1024):
            plan.spmm(B[N], C[N])
    A.bcsrVal.mul_(-2.0)
    values = (values * np.float16(-2)).astype(np.float16)
    graph.replay()
    torch.cuda.synchronize()
    for N in (16, 1024):
        check(N, C[N].data.cpu().numpy(), values)
    del graph
    plan.close()


@pytest.mark.parametrize("hint,Mb,Kb", [(8, 240, 300), (64, 240, 300), (16, 520, 700)])  # beside it a 16-row plan; a tall one
def test_both_walk_orders_of_a_range(hint, Mb, Kb):
    """A plan with two walk orders for block-rows [37, Mb - 10) of a matrix with empty block-rows and block columns in any order:
    the places of the blocks are counted from the range's first block; new values reach both copies."""
    rng = np.random.default_rng(hint)
    b0, b1 = 37, Mb - 10
    counts = rng.binomial(Kb, 0.3, Mb)
    counts[[0, 40, 41, 100, b1 - 1]] = 0
    brp, bci, bv = _blocks(rng, counts, Kb)
    order = np.concatenate([rng.permutation(np.arange(brp[r], brp[r + 1])) for r in range(Mb)])
    M, K, rows = Mb * 16, Kb * 16, (b1 - b0) * 16
    A = S.SparseMatrix.from_bcsr(M, K, brp, bci[order], bv.reshape(-1, 256)[order].reshape(-1))
    plan = S.Plan(A, b0, b1, n_hint=hint)
    assert plan.info()["kernel"] == "spmm_bcsr_stream_kernel"
    B_nk = rng.standard_normal((1032, K)).astype(np.float16)
    values = bv
    for scale in (1.0, -2.0):
        if scale != 1.0:
            A.bcsrVal.mul_(scale)
            plan.set_values()
            values = (values * np.float16(scale)).astype(np.float16)
        for N in (8, hint, 72, 1032):
            C = S.Matrix(rows, N, fill=float("nan"))
            before = S.launch_count()
            plan.spmm(S.Matrix.from_host(B_nk[:N]), C, check=True)
            assert S.launch_count() - before <= 2
            got, n0 = C.data.cpu().numpy(), max(0, N - 40)
            ref = oracle.bcsr_spmm(values, brp, bci, B_nk[n0:N], M, N - n0, K, b0, b1, threads=8).astype(np.float16).astype(np.float32)
            mag = oracle.bcsr_spmm(np.abs(values), brp, bci, np.abs(B_nk[n0:N]), M, N - n0, K, b0, b1, threads=8)
            assert float(np.max(np.abs(got[:, n0:].astype(np.float32) - ref) / (np.maximum(np.abs(ref), 1e-2 * mag) + 1e-30))) <= TOL
            assert np.all(got.reshape(b1 - b0, -1)[counts[b0:b1] == 0] == 0)
    plan.close()
