"""The tall kernel's ring of blocks and its MMA lists: steps from one block to as many as a step holds, pairs that go around the
end of the ring, lists of 0 to 16 MMAs a warp."""
import os

import numpy as np
import pytest

import oracle
import smat_b200 as S

pytestmark = pytest.mark.gpu


def _product(brp, bci, bv, B, M, N, K, rows):
    A = S.SparseMatrix.from_bcsr(M, K, brp, bci, bv)
    C = S.Matrix(M, N, fill=float("nan"))
    before = os.environ.get("SMAT_TALL_ROWS")
    os.environ["SMAT_TALL_ROWS"] = str(rows)
    S.set_variant(4)
    try:
        plan = S.Plan(A, n_hint=N)
        assert plan.info()["tall"] and plan.info()["rows_per_item"] == rows
        plan.spmm(S.Matrix.from_host(B), C, check=True)
        first = C.data.cpu().numpy().copy()
        C.data.fill_(float("nan"))
        plan.spmm(S.Matrix.from_host(B), C, check=True)
        plan.close()
    finally:
        S.set_variant(0)
        if before is None:
            del os.environ["SMAT_TALL_ROWS"]
        else:
            os.environ["SMAT_TALL_ROWS"] = before
    assert np.array_equal(first.view(np.uint16), C.data.cpu().numpy().view(np.uint16))
    return first


@pytest.mark.parametrize("rows", [1, 12, 13, 16, 19, 24])
@pytest.mark.parametrize("fill", [0.02, 0.35, 0.9, 1.0])
def test_ring_and_lists(rows, fill):
    """Twelve dense block-rows give steps of exactly 48 blocks and lists of 16 MMAs; 24 of them quads cut in two; mixed fills steps
    of all sizes, whose pairs meet the end of the ring at ever other places; one column of C tiles whole and one cut."""
    rng = np.random.default_rng(int(rows * 100 + fill * 50))
    Mb, Kb, N = 2 * rows + 1, 203, 136
    mask = rng.random((Mb, Kb)) < fill
    mask[:, ::7] &= rng.random((Mb, 29)) < 0.5 if fill < 1.0 else True
    if fill < 0.1:
        mask[Mb // 2, :] = False  # an empty block-row
    brp = np.zeros(Mb + 1, np.int32)
    brp[1:] = np.cumsum(mask.sum(axis=1))
    bci = (np.nonzero(mask)[1] * 16).astype(np.int32)
    bv = (rng.standard_normal(brp[-1] * 256) * 0.25).astype(np.float16)
    B = rng.standard_normal((N, Kb * 16)).astype(np.float16)
    C = _product(brp, bci, bv, B, Mb * 16, N, Kb * 16, rows)
    ref = oracle.bcsr_spmm(bv, brp, bci, B, Mb * 16, N, Kb * 16, threads=8)
    size = oracle.bcsr_spmm(np.abs(bv), brp, bci, np.abs(B), Mb * 16, N, Kb * 16, threads=8)
    # fp16 products are exact in fp32; both sides add at most Kb * 16 of them in fp32, in different orders (2^-24 of the sum of
    # magnitudes per addition, each), and both are rounded to fp16 (2^-11 of the value, 2^-25 below the normal range)
    bound = 2 * Kb * 16 * 2.0 ** -24 * size + 2 * 2.0 ** -11 * np.abs(ref) + 2.0 ** -24
    assert np.all(np.abs(C.astype(np.float32) - ref) <= bound)


@pytest.mark.parametrize("rows,fill", [(12, 0.45), (12, 0.6), (16, 0.36), (16, 0.42), (20, 0.28), (20, 0.34), (24, 0.23), (24, 0.28)])
def test_both_splits_of_shared_memory(rows, fill):
    """Blocks a step just below and above the line from which panels get fewer slots and the ring more blocks, over many turns of
    either ring."""
    rng = np.random.default_rng(int(rows * 1000 + fill * 100))
    Mb, Kb, N = 2 * rows, 600, 136
    mask = rng.random((Mb, Kb)) < fill
    mask[:, 100:140] = rng.random((Mb, 40)) < 0.05
    brp = np.zeros(Mb + 1, np.int32)
    brp[1:] = np.cumsum(mask.sum(axis=1))
    bci = (np.nonzero(mask)[1] * 16).astype(np.int32)
    bv = (rng.standard_normal(brp[-1] * 256) * 0.25).astype(np.float16)
    B = rng.standard_normal((N, Kb * 16)).astype(np.float16)
    C = _product(brp, bci, bv, B, Mb * 16, N, Kb * 16, rows)
    ref = oracle.bcsr_spmm(bv, brp, bci, B, Mb * 16, N, Kb * 16, threads=8)
    size = oracle.bcsr_spmm(np.abs(bv), brp, bci, np.abs(B), Mb * 16, N, Kb * 16, threads=8)
    bound = 2 * Kb * 16 * 2.0 ** -24 * size + 2 * 2.0 ** -11 * np.abs(ref) + 2.0 ** -24  # as above
    assert np.all(np.abs(C.astype(np.float32) - ref) <= bound)


@pytest.mark.parametrize("rows,fill", [(16, 0.1), (24, 0.35), (24, 0.9)])
def test_waits_that_run_out_end_the_product_and_are_reported(rows, fill):
    """The waits for blocks run out before the first list has arrived: no MMA takes its operands from shared memory that nothing was
    written to, the kernel ends, the status says so once, and the plan's next products are the one before."""
    rng = np.random.default_rng(rows)
    Mb, Kb, N = 4 * rows, 120, 264
    mask = rng.random((Mb, Kb)) < fill
    brp = np.zeros(Mb + 1, np.int32)
    brp[1:] = np.cumsum(mask.sum(axis=1))
    bci = (np.nonzero(mask)[1] * 16).astype(np.int32)
    bv = (rng.standard_normal(brp[-1] * 256) * 0.25).astype(np.float16)
    S.set_variant(4)
    try:
        plan = S.Plan(S.SparseMatrix.from_bcsr(Mb * 16, Kb * 16, brp, bci, bv), n_hint=N)
    finally:
        S.set_variant(0)
    assert plan.info()["tall"]
    Bd, C = S.Matrix.from_host(rng.standard_normal((N, Kb * 16)).astype(np.float16)), S.Matrix(Mb * 16, N, fill=float("nan"))
    plan.spmm(Bd, C, check=True)
    before = C.data.cpu().numpy().copy()
    assert S.lib().smat_selftest_plan_wait_timeout(plan._h, Bd.data.data_ptr(), C.data.data_ptr(), N, None) == 0
    assert S.lib().smat_device_status(None) == -3
    for _ in range(3):
        C.data.fill_(float("nan"))
        plan.spmm(Bd, C, check=True)
        assert np.array_equal(before.view(np.uint16), C.data.cpu().numpy().view(np.uint16))
    plan.close()
