"""Edges of the plan builder's and the launchers' choices: windows of block-columns, low tall groups, column chunks of the
host-buffer product, value updates of a range -- each against the CPU oracle; what every route refuses."""
import numpy as np
import pytest

import oracle
import smat_b200 as S

pytestmark = pytest.mark.gpu
TOL = 1e-2


def _problem(seed, Mb, Kb, N, most):
    rng = np.random.default_rng(seed)
    counts = rng.integers(1, most + 1, Mb)
    brp = np.zeros(Mb + 1, np.int32)
    brp[1:] = np.cumsum(counts)
    cols = [np.sort(rng.choice(Kb, c, replace=False)) for c in counts]
    for c in cols:
        c[-1] = Kb - 1  # the last block-column of the matrix, the first behind a full window
    bci = np.concatenate(cols).astype(np.int32) * 16
    bv = (rng.standard_normal(brp[-1] * 256) * 0.25).astype(np.float16)
    return brp, bci, bv, rng.standard_normal((N, Kb * 16)).astype(np.float16)


def _error(C, brp, bci, bv, B_nk, rows):
    N, K = B_nk.shape
    b0, b1 = rows
    M = (len(brp) - 1) * 16
    ref = oracle.bcsr_spmm(bv, brp, bci, B_nk, M, N, K, b0, b1, threads=8).astype(np.float16).astype(np.float32)
    mag = oracle.bcsr_spmm(np.abs(bv), brp, bci, np.abs(B_nk), M, N, K, b0, b1, threads=8)
    return float(np.max(np.abs(C.astype(np.float32) - ref) / (np.maximum(np.abs(ref), 1e-2 * mag) + 1e-30)))


@pytest.mark.parametrize("variant", [1, 4])
@pytest.mark.parametrize("Kb", [2048, 2049, 4096, 4097, 8192, 8193, 16385])
def test_windows_of_block_columns(Kb, variant):
    brp, bci, bv, B_nk = _problem(Kb, 40, Kb, 24, 60)
    A, B, C = S.SparseMatrix.from_bcsr(640, Kb * 16, brp, bci, bv), S.Matrix.from_host(B_nk), S.Matrix(640, 24, fill=float("nan"))
    S.set_variant(variant)
    try:
        plan = S.Plan(A, n_hint=24)
        plan.spmm(B, C, check=True)
        assert _error(C.data.cpu().numpy(), brp, bci, bv, B_nk, (0, 40)) <= TOL
        plan.close()
        if variant == 1:  # the plan built inside a call
            C.data.fill_(float("nan"))
            S.spmm(A, B, C, check=True)
            assert _error(C.data.cpu().numpy(), brp, bci, bv, B_nk, (0, 40)) <= TOL
    finally:
        S.set_variant(0)


@pytest.mark.parametrize("height,N", [(12, 24), (14, 136), (18, 128)])
def test_low_tall_groups_and_value_update_of_a_range(height, N, monkeypatch):
    monkeypatch.setenv("SMAT_TALL_ROWS", str(height))
    brp, bci, bv, B_nk = _problem(height, 75, 130, N, 60)
    A, B = S.SparseMatrix.from_bcsr(75 * 16, 130 * 16, brp, bci, bv), S.Matrix.from_host(B_nk)
    S.set_variant(4)
    try:
        plan = S.Plan(A, 7, 70, n_hint=N)
    finally:
        S.set_variant(0)
    assert plan.info()["tall"] and plan.info()["rows_per_item"] == height
    A.bcsrVal.mul_(-2.0)
    plan.set_values()
    C = S.Matrix(63 * 16, N, fill=float("nan"))
    plan.spmm(B, C, check=True)
    plan.close()
    assert _error(C.data.cpu().numpy(), brp, bci, (bv * np.float16(-2)).astype(np.float16), B_nk, (7, 70)) <= TOL


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("N", [8, 64, 72, 200, 520])
def test_host_buffers_by_column_chunks(N, pinned):
    """Pinned C: columns go out chunk by chunk (the last one halved); pageable C: whole rows by the copy engine."""
    import torch
    brp, bci, bv, B_nk = _problem(N, 50, 90, N, 30)
    plan = S.Plan(S.SparseMatrix.from_bcsr(800, 1440, brp, bci, bv), n_hint=N)
    B_host, C_host = torch.from_numpy(B_nk.view(np.int16)), torch.full((800, N), -1, dtype=torch.int16)
    if pinned:
        B_host, C_host = B_host.pin_memory(), C_host.pin_memory()
    for _ in range(2):
        C_host.fill_(-1)
        plan.spmm_host(B_host, C_host)
        torch.cuda.synchronize()
        assert _error(C_host.numpy().view(np.float16), brp, bci, bv, B_nk, (0, 50)) <= TOL
    plan.close()


def test_part_of_a_pinned_buffer_is_stored_to_by_the_kernels():
    """C inside a larger pinned allocation goes out by columns (a store kernel per chunk), as a whole allocation does; the
    same buffer in pageable memory takes no such kernel."""
    import torch
    brp, bci, bv, B_nk = _problem(11, 50, 90, 200, 30)
    plan = S.Plan(S.SparseMatrix.from_bcsr(800, 1440, brp, bci, bv), n_hint=200)
    B_host = torch.from_numpy(B_nk.view(np.int16)).pin_memory()
    launches = {}
    for name, flat in (("pinned", torch.empty(800 * 200 + 4096, dtype=torch.int16).pin_memory()),
                       ("pageable", torch.empty(800 * 200 + 4096, dtype=torch.int16))):
        C_host = flat[2048:2048 + 800 * 200].view(800, 200)
        flat.fill_(-1)
        before = S.launch_count()
        plan.spmm_host(B_host, C_host)
        torch.cuda.synchronize()
        launches[name] = S.launch_count() - before
        assert _error(C_host.numpy().view(np.float16), brp, bci, bv, B_nk, (0, 50)) <= TOL
        assert bool((flat[:2048] == -1).all()) and bool((flat[2048 + 800 * 200:] == -1).all())
    plan.close()
    assert launches["pinned"] >= 4 and launches["pinned"] > launches["pageable"]


# (variant, entry): the kernels that see the boundary's arrays first -- plan kernels of both walk orders, stream kernel
ROUTES = [(0, "call"), (1, "call"), (5, "call"), (1, "static"), (5, "static"), (0, "plan"), (1, "plan"), (4, "plan"), (5, "plan")]


def _status_of(route, A, B, C):
    import torch
    variant, entry = route
    L, stream, (N, K) = S.lib(), torch.cuda.current_stream().cuda_stream, B.data.shape
    S.set_variant(variant)
    try:
        if entry == "plan":
            plan = S.Plan(A, n_hint=N)
            plan.spmm(B, C)
            rc, text = L.smat_device_status(stream), L.smat_last_error_string()
            plan.close()
        else:
            S.spmm(A, B, C) if entry == "call" else S.api._check(L.smat_spmm_bcsr_f16_static(
                A.getBcsrValues(), A.getBcsrRowPtr(), A.getBcsrColIdx(), B.data.data_ptr(), C.data.data_ptr(), A.M, N, K, A.nnzb, stream))
            rc, text = L.smat_device_status(stream), L.smat_last_error_string()
    finally:
        S.set_variant(0)
    assert L.smat_device_status(stream) == 0
    return rc, b"ascending" in text


@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("late,early", [(1, 1), (40, 1), (300, 3)])
def test_block_columns_out_of_order_are_reported_by_every_kernel(route, late, early):
    """A block-row whose first `late` blocks lie in the second window of 16384 block-columns and whose next `early` ones in
    the first: within 32 columns read together, across two such batches, across the warps and pieces of a long row."""
    Kb, N = 20000, 16
    good = np.sort(np.random.default_rng(late).choice(Kb, 9, replace=False))
    cols = [good, np.concatenate([16384 + 7 * np.arange(late), 5 + np.arange(early)]), good]
    brp = np.cumsum([0] + [len(c) for c in cols]).astype(np.int32)
    bci = (np.concatenate(cols) * 16).astype(np.int32)
    A = S.SparseMatrix.from_bcsr(48, Kb * 16, brp, bci, np.ones(brp[-1] * 256, np.float16))
    B, C = S.Matrix(N, Kb * 16, fill=1.0), S.Matrix(48, N, fill=0.0)
    assert _status_of(route, A, B, C) == (-6, True)


@pytest.mark.parametrize("route", ROUTES)
def test_order_inside_a_window_does_not_matter(route):
    rng = np.random.default_rng(8)
    brp, bci, bv, B_nk = _problem(3, 40, 700, 16, 60)
    order = np.concatenate([rng.permutation(np.arange(brp[r], brp[r + 1])) for r in range(40)])
    A = S.SparseMatrix.from_bcsr(640, 11200, brp, bci[order], bv.reshape(-1, 256)[order].reshape(-1))
    C = S.Matrix(640, 16, fill=float("nan"))
    assert _status_of(route, A, S.Matrix.from_host(B_nk), C) == (0, False)
    assert _error(C.data.cpu().numpy(), brp, bci, bv, B_nk, (0, 40)) <= TOL


@pytest.mark.parametrize("N,tall", [(256, False), (1024, True)])
def test_plan_of_few_blocks_a_step_is_tall_only_where_that_is_faster(N, tall):
    """Some 105 000 scattered blocks, six of them a step: one round of items either way at 256 columns, which the 16-row kernel takes 63 us
    for and the tall kernel 68; several at 1024 (228 and 173)."""
    rng = np.random.default_rng(1)
    mask = rng.random((1024, 1024)) < 0.1
    brp = np.zeros(1025, np.int32)
    brp[1:] = np.cumsum(mask.sum(axis=1))
    A = S.SparseMatrix.from_bcsr(16384, 16384, brp, (np.nonzero(mask)[1] * 16).astype(np.int32), np.zeros(brp[-1] * 256, np.float16))
    plan = S.Plan(A, n_hint=N)
    assert plan.info()["tall"] == tall
    plan.close()
