"""Wide products of the stream kernels from slabs, whose slices come through a ring in shared memory: block-rows shorter than the
ring, empty ones, one, two and four warps a block-row, long block-rows in pieces, tiles of every width class and their edges, with a
plan and without."""
import threading

import numpy as np
import pytest
import torch

import oracle
import smat_b200 as S

pytestmark = pytest.mark.gpu


def _matrix(rng, Mb, Kb, most, long_row=None):
    counts = rng.integers(0, most + 1, Mb)
    counts[:6] = [0, 1, 2, 3, 4, min(5, Kb)]  # shorter than the ring, as long, one longer
    if long_row is not None:
        counts[long_row] = Kb
    cols = [np.sort(rng.choice(Kb, c, replace=False)) for c in counts]
    brp = np.zeros(Mb + 1, np.int32)
    brp[1:] = np.cumsum(counts)
    return brp, (np.concatenate(cols) * 16).astype(np.int32), (rng.standard_normal(brp[-1] * 256) * 0.25).astype(np.float16)


@pytest.mark.parametrize("plan", [True, False])
@pytest.mark.parametrize("Mb,Kb,most,long_row", [(2400, 300, 40, None), (1100, 260, 60, 7), (300, 700, 300, 11)])
@pytest.mark.parametrize("N", [40, 64, 72, 96, 104, 128, 136, 200])
def test_ring_against_oracle(plan, Mb, Kb, most, long_row, N):
    rng = np.random.default_rng(N + Mb)
    M, K = Mb * 16, Kb * 16
    brp, bci, bv = _matrix(rng, Mb, Kb, most, long_row)
    B = rng.standard_normal((N, K)).astype(np.float16)
    A = S.SparseMatrix.from_bcsr(M, K, brp, bci, bv)
    Bd, C = S.Matrix.from_host(B), S.Matrix(M, N, fill=float("nan"))
    outs = []
    S.set_variant(5)
    try:
        p = S.Plan(A, n_hint=N) if plan else None
        for _ in range(2):
            C.data.fill_(float("nan"))
            p.spmm(Bd, C, check=True) if plan else S.spmm(A, Bd, C, check=True)
            outs.append(C.data.cpu().numpy().copy())
        if plan:
            p.close()
    finally:
        S.set_variant(0)
    assert np.array_equal(outs[0].view(np.uint16), outs[1].view(np.uint16))
    ref = oracle.bcsr_spmm(bv, brp, bci, B, M, N, K, threads=8)
    size = oracle.bcsr_spmm(np.abs(bv), brp, bci, np.abs(B), M, N, K, threads=8)
    # exact products, at most K additions in fp32 on either side (2^-24 of the sum of magnitudes each), one rounding to fp16 each
    bound = 2 * K * 2.0 ** -24 * size + 2 * 2.0 ** -11 * np.abs(ref) + 2.0 ** -24
    assert np.all(np.abs(outs[0].astype(np.float32) - ref) <= bound)


@pytest.mark.parametrize("plan", [True, False])
@pytest.mark.parametrize("Mb,Kb,most,blocks", [(2400, 300, 30, (32768, 65536)), (2400, 300, 60, (65536, 1 << 30)), (300, 2400, 260, (32768, 65536))])
@pytest.mark.parametrize("N", [40, 64])
def test_both_kernels_of_33_to_64_columns(plan, Mb, Kb, most, blocks, N):
    """From slabs, with the loads in registers (without a plan; with one between 32768 and 65536 blocks) and through the ring, one and
    four warps a block-row; beyond 4.5 MB of slabs (Kb = 2400, 64 columns) all through the ring."""
    rng = np.random.default_rng(Mb + most + N)
    M, K = Mb * 16, Kb * 16
    brp, bci, bv = _matrix(rng, Mb, Kb, most)
    assert blocks[0] <= brp[-1] < blocks[1]
    B = rng.standard_normal((N, K)).astype(np.float16)
    A, Bd, C = S.SparseMatrix.from_bcsr(M, K, brp, bci, bv), S.Matrix.from_host(B), S.Matrix(M, N, fill=float("nan"))
    S.set_variant(5)
    try:
        if plan:
            p = S.Plan(A, n_hint=N)
            p.spmm(Bd, C, check=True)
            p.close()
        else:
            S.spmm(A, Bd, C, check=True)
    finally:
        S.set_variant(0)
    ref = oracle.bcsr_spmm(bv, brp, bci, B, M, N, K, threads=8)
    size = oracle.bcsr_spmm(np.abs(bv), brp, bci, np.abs(B), M, N, K, threads=8)
    bound = 2 * K * 2.0 ** -24 * size + 2 * 2.0 ** -11 * np.abs(ref) + 2.0 ** -24  # as above
    assert np.all(np.abs(C.data.cpu().numpy().astype(np.float32) - ref) <= bound)


def test_ring_skips_columns_outside_the_matrix():
    """A block whose column lies outside the matrix is left out and reported, with the ring as with the other kernels."""
    rng = np.random.default_rng(3)
    Mb, Kb, N = 2400, 300, 128
    M, K = Mb * 16, Kb * 16
    brp, bci, bv = _matrix(rng, Mb, Kb, 40)
    B = rng.standard_normal((N, K)).astype(np.float16)
    row = int(np.argmax(np.diff(brp)))
    bad, good = bci.copy(), bv.copy()
    bad[brp[row + 1] - 1] = K
    good[(brp[row + 1] - 1) * 256: brp[row + 1] * 256] = 0
    C = S.Matrix(M, N, fill=float("nan"))
    S.set_variant(5)
    try:
        with pytest.raises(S.SmatError):
            S.spmm(S.SparseMatrix.from_bcsr(M, K, brp, bad, bv), S.Matrix.from_host(B), C, check=True)
        got = C.data.cpu().numpy().copy()
        S.spmm(S.SparseMatrix.from_bcsr(M, K, brp, bci, good), S.Matrix.from_host(B), C, check=True)
    finally:
        S.set_variant(0)
    # another order of nothing but a block of zeros: the same sums
    assert np.array_equal(got.view(np.uint16), C.data.cpu().numpy().view(np.uint16))


@pytest.mark.parametrize("Mb,Kb,most,long_row,N", [(2400, 300, 40, None, 128), (2400, 300, 40, None, 96), (1100, 260, 60, None, 128),
                                                   (300, 700, 300, None, 128), (2400, 300, 40, 7, 128), (1100, 600, 60, 9, 128)])
def test_waits_that_run_out_end_the_product_and_are_reported(Mb, Kb, most, long_row, N):
    """One, two and four warps a block-row give up their first wait (all lanes of a warp, and all warps reach the sum of a block-row):
    the kernel ends, the status says so once, and the plan's next products are the one before, of long block-rows too, whose pieces
    are counted as they arrive."""
    rng = np.random.default_rng(N)
    M, K = Mb * 16, Kb * 16
    brp, bci, bv = _matrix(rng, Mb, Kb, most, long_row)
    Bd, C = S.Matrix.from_host(rng.standard_normal((N, K)).astype(np.float16)), S.Matrix(M, N, fill=float("nan"))
    S.set_variant(5)
    try:
        p = S.Plan(S.SparseMatrix.from_bcsr(M, K, brp, bci, bv), n_hint=N)
    finally:
        S.set_variant(0)
    p.spmm(Bd, C, check=True)
    before = C.data.cpu().numpy().copy()
    assert S.lib().smat_selftest_plan_wait_timeout(p._h, Bd.data.data_ptr(), C.data.data_ptr(), N, None) == 0
    assert S.lib().smat_device_status(None) == -3 and b"site code 40" in S.lib().smat_last_error_string()
    for _ in range(3):
        C.data.fill_(float("nan"))
        p.spmm(Bd, C, check=True)
        assert np.array_equal(before.view(np.uint16), C.data.cpu().numpy().view(np.uint16))
    p.close()


@pytest.mark.parametrize("N", [112, 120, 128])
def test_block_rows_that_take_fewer_warps(N):
    """Some 60 blocks a block-row and more than one round of warps: 12 warps an SM from 113 columns on."""
    rng = np.random.default_rng(N)
    Mb, Kb = 2400, 300
    M, K = Mb * 16, Kb * 16
    brp, bci, bv = _matrix(rng, Mb, Kb, 120)
    B = rng.standard_normal((N, K)).astype(np.float16)
    A, Bd, C = S.SparseMatrix.from_bcsr(M, K, brp, bci, bv), S.Matrix.from_host(B), S.Matrix(M, N, fill=float("nan"))
    S.set_variant(5)
    try:
        p = S.Plan(A, n_hint=N)
    finally:
        S.set_variant(0)
    p.spmm(Bd, C, check=True)
    p.close()
    got = C.data.cpu().numpy().astype(np.float32)
    assert np.all(np.isfinite(got))
    for b0 in (0, 1000, Mb - 200):
        ref = oracle.bcsr_spmm(bv, brp, bci, B, M, N, K, b0, b0 + 200, threads=8)
        size = oracle.bcsr_spmm(np.abs(bv), brp, bci, np.abs(B), M, N, K, b0, b0 + 200, threads=8)
        bound = 2 * K * 2.0 ** -24 * size + 2 * 2.0 ** -11 * np.abs(ref) + 2.0 ** -24  # as above
        assert np.all(np.abs(got[b0 * 16: (b0 + 200) * 16] - ref) <= bound)


def test_small_and_large_slabs_from_two_threads():
    """Slabs of more than half of L2 are multiplied by the same kernel with more shared memory for each CTA: two threads that launch
    it so and so do not refuse each other's launch, and both products are right."""
    N, plans = 128, []
    for Mb, Kb, most in [(2400, 16384, 120), (2400, 300, 40)]:  # 67 MB of slabs, 1.2 MB
        rng = np.random.default_rng(Kb)
        M, K = Mb * 16, Kb * 16
        brp, bci, bv = _matrix(rng, Mb, Kb, most)
        B = rng.standard_normal((N, K)).astype(np.float16)
        A, Bd, C = S.SparseMatrix.from_bcsr(M, K, brp, bci, bv), S.Matrix.from_host(B), S.Matrix(M, N, fill=float("nan"))
        S.set_variant(5)
        try:
            plan = S.Plan(A, n_hint=N)
        finally:
            S.set_variant(0)
        plan.spmm(Bd, C, check=True)
        ref = oracle.bcsr_spmm(bv, brp, bci, B, M, N, K, threads=8)
        size = oracle.bcsr_spmm(np.abs(bv), brp, bci, np.abs(B), M, N, K, threads=8)
        bound = 2 * K * 2.0 ** -24 * size + 2 * 2.0 ** -11 * np.abs(ref) + 2.0 ** -24  # as above
        assert np.all(np.abs(C.data.cpu().numpy().astype(np.float32) - ref) <= bound)
        plans.append((plan, Bd, C, C.data.clone()))
    errors, start = [], threading.Barrier(2)

    def work(plan, Bd, C, first):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for _ in range(300):
                    plan.spmm(Bd, C)
                torch.cuda.current_stream().synchronize()
            assert torch.equal(C.data, first)
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=p) for p in plans]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert S.lib().smat_device_status(None) == 0
