"""Edges of the plan builder's and the launchers' choices: windows of block-columns, low tall groups, column chunks of the
host-buffer product, value updates of a range -- each against the CPU oracle."""
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
