"""Products without a plan on the tcgen05 kernel: blocks gathered from the boundary's array.  The same plan with a packed copy has the
same blocks in the same places; a range of block-rows, steps of one to 24 blocks, quads cut in
several steps, an empty block-row, columns that do not fill a quad, narrow and several tiles of C."""
import numpy as np
import pytest
import torch

import oracle
import smat_b200 as S

pytestmark = pytest.mark.gpu


def _matrix(rng, Mb, Kb, fill):
    mask = rng.random((Mb, Kb)) < fill
    mask[Mb // 2] = False
    mask[:3, :8] = True
    brp = np.zeros(Mb + 1, np.int32)
    brp[1:] = np.cumsum(mask.sum(axis=1))
    return brp, (np.nonzero(mask)[1] * 16).astype(np.int32), (rng.standard_normal(brp[-1] * 256) * 0.25).astype(np.float16)


@pytest.mark.parametrize("Mb,Kb,fill", [(1, 9, 0.3), (33, 70, 0.02), (70, 131, 0.35), (40, 333, 1.0), (300, 41, 0.2)])
@pytest.mark.parametrize("N", [8, 120, 128, 264])
def test_gather_against_oracle_and_packed(Mb, Kb, fill, N):
    rng = np.random.default_rng(Mb * 7 + N)
    M, K = Mb * 16, Kb * 16
    brp, bci, bv = _matrix(rng, Mb, Kb, fill)
    B = rng.standard_normal((N, K)).astype(np.float16)
    A, Bd = S.SparseMatrix.from_bcsr(M, K, brp, bci, bv), S.Matrix.from_host(B)
    ref = oracle.bcsr_spmm(bv, brp, bci, B, M, N, K, threads=8)
    size = oracle.bcsr_spmm(np.abs(bv), brp, bci, np.abs(B), M, N, K, threads=8)
    # exact products, at most K additions in fp32 on either side (2^-24 of the sum of magnitudes each), one rounding to fp16 each
    bound = 2 * K * 2.0 ** -24 * size + 2 * 2.0 ** -11 * np.abs(ref) + 2.0 ** -24
    C, first = S.Matrix(M, N, fill=float("nan")), Mb // 3
    shard = S.Matrix(M - first * 16, N, fill=float("nan"))
    S.set_variant(1)
    try:
        S.spmm(A, Bd, C, check=True)
        S.spmm_rows(A, Bd, shard, first, Mb, check=True)
    finally:
        S.set_variant(0)
    got = C.data.cpu().numpy()
    assert np.all(np.abs(got.astype(np.float32) - ref) <= bound)
    assert np.all(np.abs(shard.data.cpu().numpy().astype(np.float32) - ref[first * 16:]) <= bound[first * 16:])
    packed = S.Matrix(M, N, fill=float("nan"))
    S.set_variant(2)  # reads a packed copy
    try:
        S.spmm(A, Bd, packed, check=True)
    finally:
        S.set_variant(0)
    assert torch.all((packed.data.float() - C.data.float()).abs() <= torch.from_numpy(2 * bound).cuda())


@pytest.mark.parametrize("call", ["spmm", "static"])
@pytest.mark.parametrize("Mb,Kb,fill,N,packed", [(2048, 70, 0.2, 1536, False), (2048, 70, 0.2, 1544, True), (2048, 20, 0.2, 1544, False),
                                                 (512, 70, 0.4, 3072, False), (512, 70, 0.4, 3080, True), (511, 70, 0.4, 3080, False)])
def test_wide_products_read_a_packed_copy(call, Mb, Kb, fill, N, packed):
    """Many tiles of C, block-rows and blocks: the blocks are copied into walk order first (three launches more), else they are
    gathered; either way the product is the oracle's."""
    rng = np.random.default_rng(Kb + N)
    M, K = Mb * 16, Kb * 16
    brp, bci, bv = _matrix(rng, Mb, Kb, fill)
    B = rng.standard_normal((N, K)).astype(np.float16)
    A, Bd, C = S.SparseMatrix.from_bcsr(M, K, brp, bci, bv), S.Matrix.from_host(B), S.Matrix(M, N, fill=float("nan"))
    S.set_variant(1)
    before = S.launch_count()
    try:
        if call == "spmm":
            S.spmm(A, Bd, C)
        else:
            assert S.lib().smat_spmm_bcsr_f16_static(A.getBcsrValues(), A.getBcsrRowPtr(), A.getBcsrColIdx(), Bd.data.data_ptr(),
                                                     C.data.data_ptr(), M, N, K, A.nnzb, None) == 0
    finally:
        S.set_variant(0)
    assert S.lib().smat_device_status(None) == 0
    assert (S.launch_count() - before >= 5) == packed
    got = C.data.cpu().numpy().astype(np.float32)
    assert np.all(np.isfinite(got))
    for b0 in (0, Mb // 2 - 4, Mb - 8):
        ref = oracle.bcsr_spmm(bv, brp, bci, B, M, N, K, b0, b0 + 8, threads=8)
        size = oracle.bcsr_spmm(np.abs(bv), brp, bci, np.abs(B), M, N, K, b0, b0 + 8, threads=8)
        bound = 2 * K * 2.0 ** -24 * size + 2 * 2.0 ** -11 * np.abs(ref) + 2.0 ** -24  # as above
        assert np.all(np.abs(got[b0 * 16: b0 * 16 + 128] - ref) <= bound)


@pytest.mark.parametrize("what", ["column", "order", "rowptr", "dip"])
def test_gather_reports_inconsistent_arrays(what):
    """Columns outside the matrix, block columns that go back to an earlier window, row pointers beyond the blocks or that go down so
    that a block-row claims others' blocks, more than its group has room for: reported, and the next product is right."""
    rng = np.random.default_rng(9)
    Mb, Kb, N = 20, 17000, 128
    M, K = Mb * 16, Kb * 16
    brp, bci, bv = _matrix(rng, Mb, Kb, 0.002)
    B = rng.standard_normal((N, K)).astype(np.float16)
    row = 5
    bad_rp, bad_ci = brp.copy(), bci.copy()
    if what == "column":
        bad_ci[brp[row + 1] - 1] = K
    elif what == "order":
        bad_ci[brp[row]] = K - 16
    elif what == "rowptr":
        bad_rp[-1] = brp[-1] + 5
    else:
        bad_rp[row + 1] = brp[row - 3]
    Bd, C = S.Matrix.from_host(B), S.Matrix(M, N, fill=float("nan"))
    S.set_variant(1)
    try:
        with pytest.raises(S.SmatError):
            S.spmm(S.SparseMatrix.from_bcsr(M, K, bad_rp, bad_ci, bv), Bd, C, check=True)
        S.spmm(S.SparseMatrix.from_bcsr(M, K, brp, bci, bv), Bd, C, check=True)
    finally:
        S.set_variant(0)
    ref = oracle.bcsr_spmm(bv, brp, bci, B, M, N, K, threads=8)
    assert np.allclose(C.data.cpu().numpy().astype(np.float32), ref, rtol=2e-3, atol=2e-3 * np.abs(ref).max())
