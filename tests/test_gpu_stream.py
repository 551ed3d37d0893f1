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


def _multiply(brp, bci, bv, B_nk, M, K, plan):
    N = B_nk.shape[0]
    A, B, C = S.SparseMatrix.from_bcsr(M, K, brp, bci, bv), S.Matrix.from_host(B_nk), S.Matrix(M, N, fill=float("nan"))
    S.set_variant(5)
    try:
        if plan:
            p = S.Plan(A, n_hint=min(N, 136))  # wider products than the hint go in several passes
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
