"""Cases on which the speed of this framework is measured: what a user has it do, through its public entry points.

A case is one call pattern ("entry") on one kind of matrix ("matrix") at one size.

Entries
  plan    a program that multiplies one sparse matrix many times: `Plan` once, `Plan.spmm` per pass (serving, solvers)
  call    a program that keeps no plan: `spmm` straight from the blocked arrays, the signature of the launcher that the
          framework stands in for; everything the product needs is worked out inside the call
  update  the values of the matrix change between products (training of a pruned layer): `Plan.set_values`, `Plan.spmm`
  block   host CSR -> blocked matrix on the device: `SparseMatrix.from_csr`, which starts on host arrays by its nature
  host    B and C live in pinned host memory: `Plan.spmm_host`, with the copies in and out

Matrices (the five benchmark configurations, and sizes around them)
  band        all entries with |i - j| <= half_bandwidth (banded solvers); blocks lie side by side around the diagonal
  layer       weight matrix of which a share `fill` of the 16 x 16 blocks is kept at random, each kept block dense; N is the
              number of activation columns: a few when decoding, thousands when a prompt or a batch is processed
  uniform     entries at random positions: most blocks hold one or two entries
  powerlaw    graph with Zipf degrees and 70 % of the targets near the row; rows in the given order or sorted by degree
              (a cheap reorder; like the similarity reorder it gathers the heavy rows in a few block-rows)
  clustered   256 x 256 clusters near the diagonal at 30 % fill, and a few stray entries (finite elements)
"""
import math

import numpy as np
import torch

import smat_b200 as S


def listed():
    return [
        # The smallest calls: a small banded system with a narrow B.  Latency, launches and host work decide.
        {"name": "band_plan", "entry": "plan", "matrix": "band", "M": 4096, "K": 4096, "half_bandwidth": 64, "N": 64},
        # The same kind of system without a plan, at an odd size and width: what one stand-alone call costs.
        {"name": "band_call", "entry": "call", "matrix": "band", "M": 2288, "K": 2288, "half_bandwidth": 40, "N": 72},
        # Decoding with a pruned layer: all weights are read for a handful of activation columns.
        {"name": "layer_decode", "entry": "plan", "matrix": "layer", "M": 8192, "K": 28672, "fill": 0.2, "N": 16},
        # The same layer on a prompt of 4096 columns (the benchmark's default workload).
        {"name": "layer_prefill", "entry": "plan", "matrix": "layer", "M": 8192, "K": 28672, "fill": 0.2, "N": 4096},
        # A smaller layer whose sizes divide nothing, with a batch in between.
        {"name": "layer_ragged", "entry": "plan", "matrix": "layer", "M": 3056, "K": 8176, "fill": 0.35, "N": 1000},
        # Random sparse matrix: low fill inside the blocks, the largest number of blocks.
        {"name": "uniform", "entry": "plan", "matrix": "uniform", "M": 65536, "K": 65536, "density": 0.001, "N": 256},
        # Graph: scattered blocks, a few block-rows many times heavier than the rest.
        {"name": "powerlaw", "entry": "plan", "matrix": "powerlaw", "M": 262144, "K": 262144, "order": "degree", "N": 128},
        # Finite elements: dense clusters, the largest matrix and the largest B and C.
        {"name": "clustered", "entry": "plan", "matrix": "clustered", "M": 524288, "K": 524288, "N": 512},
        # A stand-alone call on a mid-size random matrix: the plan inside the call is most of the work.
        {"name": "uniform_call", "entry": "call", "matrix": "uniform", "M": 16384, "K": 16384, "density": 0.001, "N": 256},
        # One training step's forward product of a pruned layer: new values, then the product.
        {"name": "layer_update", "entry": "update", "matrix": "layer", "M": 4096, "K": 4096, "fill": 0.25, "N": 512},
        # A graph arrives as CSR on the host and is blocked on the device.
        {"name": "powerlaw_block", "entry": "block", "matrix": "powerlaw", "M": 65536, "K": 65536, "order": "given", "N": 0},
        # Activations come from the host and results go back to it.
        {"name": "layer_host", "entry": "host", "matrix": "layer", "M": 4096, "K": 14336, "fill": 0.2, "N": 1024},
    ]


def _log(rng, lo, hi, multiple):
    """A multiple of `multiple` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi // multiple, max(-(-lo // multiple), round(v / multiple)))) * multiple


def draw(rng):
    entry = rng.choice(["plan", "plan", "plan", "plan", "plan", "call", "call", "update", "block", "host"])
    if entry in ("update", "host"):
        matrix = "layer"
    elif entry == "block":
        matrix = rng.choice(["uniform", "powerlaw", "clustered", "band"])
    else:
        matrix = rng.choice(["layer", "layer", "uniform", "powerlaw", "clustered", "band"])
    c = {"entry": entry, "matrix": matrix}
    small = entry in ("call", "block")
    if matrix == "band":
        c["M"] = c["K"] = _log(rng, 512, 32768, 16)
        c["half_bandwidth"] = _log(rng, 8, 256, 1)
        c["N"] = _log(rng, 8, 512, 8)
    elif matrix == "layer":
        c["M"] = _log(rng, 512, 4096 if entry != "plan" else 8192, 16)
        c["K"] = _log(rng, 512, {"plan": 28672, "host": 14336}.get(entry, 8192), 16)
        c["fill"] = round(rng.uniform(0.05, 0.2 if entry == "host" else 0.4), 3)
        c["N"] = _log(rng, 64 if entry == "host" else 8, {"plan": 4096, "host": 1024}.get(entry, 512), 8)
        most = 8192 * 28672 * 0.2  # stored values of the largest listed layer
        c["fill"] = round(min(c["fill"], most / (c["M"] * c["K"])), 3)
    elif matrix == "uniform":
        c["M"] = c["K"] = _log(rng, 2048, 16384 if small else 65536, 16)
        most = 0.001 * (16384.0 if small else 65536.0) ** 2  # entries of the largest listed matrix
        c["density"] = round(math.exp(rng.uniform(math.log(2e-4), math.log(min(4e-3, most / c["M"] ** 2)))), 6)
        c["N"] = _log(rng, 8, 256, 8)
    elif matrix == "powerlaw":
        c["M"] = c["K"] = _log(rng, 4096, 65536 if small else 262144, 16)
        c["order"] = rng.choice(["given", "degree"])
        c["N"] = _log(rng, 8, 128, 8)
    else:
        c["M"] = c["K"] = _log(rng, 4096, 65536 if small else 524288, 256)
        c["N"] = _log(rng, 8, 512, 8)
    if entry == "block":
        c["N"] = 0
    return c


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _layer(case, g):
    """The blocked arrays of a pruned layer, as a checkpoint of such weights holds them (host arrays)."""
    Mb, Kb = case["M"] // 16, case["K"] // 16
    kept = torch.rand((Mb, Kb), device="cuda", generator=g) < case["fill"]
    rowptr = torch.zeros(Mb + 1, dtype=torch.int32, device="cuda")
    rowptr[1:] = kept.sum(1).cumsum(0)
    colidx = (kept.nonzero()[:, 1] * 16).to(torch.int32)
    vals = (torch.randn(colidx.numel() * 256, device="cuda", generator=g) * 0.02).half()
    return rowptr.cpu().numpy(), colidx.cpu().numpy(), vals.cpu().numpy()


def _csr(case, g):
    """CSR on the host (columns ascending) of the matrices that are given by entries."""
    n, kind, values = case["M"], case["matrix"], g
    if case["entry"] == "block":  # so that matrices of all seeds have as many blocks: one pattern, moved along the diagonal below
        g = _generator(1)
    if kind == "band":
        b = case["half_bandwidth"]
        i = torch.arange(n, device="cuda").repeat_interleave(2 * b + 1)
        j = i + torch.arange(-b, b + 1, device="cuda").repeat(n)
        inside = (j >= 0) & (j < n)
        keys = i[inside] * n + j[inside]
    elif kind == "uniform":
        keys = torch.randint(0, n * n, (int(round(case["density"] * n * n)),), device="cuda", generator=g).unique()
    elif kind == "powerlaw":
        # degrees ~ Zipf(2.1) scaled to 16 on average, at most 8192: the inverse of the distribution's tail, cut to whole
        # numbers; 70 % of the targets within +-512 of the row, the rest anywhere
        u = torch.rand(n, device="cuda", generator=g, dtype=torch.float64).clamp_(min=1e-12)
        z = (u ** (-1.0 / 1.1)).floor().clamp_(max=8192.0)
        degree = (z * 16.0 / z.mean()).round().clamp_(1, min(8192, n)).long()
        i = torch.arange(n, device="cuda").repeat_interleave(degree)
        near = torch.rand(i.numel(), device="cuda", generator=g) < 0.7
        lo, hi = (i - 512).clamp_(min=0), (i + 512).clamp_(max=n - 1)
        local = lo + (torch.rand(i.numel(), device="cuda", generator=g, dtype=torch.float64) * (hi - lo + 1)).long()
        keys = (i * n + torch.where(near, local, torch.randint(0, n, (i.numel(),), device="cuda", generator=g))).unique()
        if case["order"] == "degree":
            place = torch.empty(n, dtype=torch.long, device="cuda")
            place[torch.bincount(keys // n, minlength=n).argsort(descending=True, stable=True)] = torch.arange(n, device="cuda")
            keys = (place[keys // n] * n + keys % n).sort().values
    else:
        clusters = n // 256
        start = 256 * torch.arange(clusters, device="cuda") + 16 * torch.randint(-16, 17, (clusters,), device="cuda", generator=g)
        start.clamp_(0, n - 256)
        c, r, k = (torch.rand((clusters, 256, 256), device="cuda", generator=g) < 0.3).nonzero(as_tuple=True)
        keys = (256 * c + r) * n + start[c] + k
        keys = torch.cat([keys, torch.randint(0, n * n, (int(1e-5 * keys.numel()) + 1,), device="cuda", generator=g)]).unique()
    if case["entry"] == "block" and kind != "band":
        by = 16 * torch.randint(0, n // 16, (1,), device="cuda", generator=values)
        keys = ((keys // n + by) % n * n + (keys % n + by) % n).sort().values
    rowptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    rowptr[1:] = torch.bincount(keys // n, minlength=n).cumsum(0)
    count, g = keys.numel(), values
    if kind == "clustered":
        vals = torch.randn(count, device="cuda", generator=g) * 0.1
    elif kind == "uniform":
        vals = torch.randn(count, device="cuda", generator=g)
    elif kind == "powerlaw":
        vals = torch.rand(count, device="cuda", generator=g)
    else:
        vals = torch.rand(count, device="cuda", generator=g) * 2 - 1
    return rowptr.cpu().numpy(), (keys % n).to(torch.int32).cpu().numpy(), vals.half().cpu().numpy()


def prepare(case, seed):
    g = _generator(seed)
    M, K, N, entry = case["M"], case["K"], case["N"], case["entry"]
    if case["matrix"] == "layer":
        A = S.SparseMatrix.from_bcsr(M, K, *_layer(case, g))
    else:
        csr = _csr(case, g)
        if entry == "block":
            return {"entry": entry, "M": M, "K": K, "csr": csr}
        A = S.SparseMatrix.from_csr(M, K, *csr)
    state = {"entry": entry, "A": A}
    if entry != "call":
        state["plan"] = S.Plan(A, n_hint=N)
    B = torch.randn((N, K), device="cuda", generator=g).half()  # column n of the K x N matrix is row n
    if entry == "host":
        state["B"] = torch.empty((N, K), dtype=torch.float16).pin_memory()
        state["B"].copy_(B)
        state["C"] = torch.empty((M, N), dtype=torch.float16).pin_memory()
    else:
        state["B"] = B
        state["C"] = torch.empty((M, N), dtype=torch.float16, device="cuda")
    return state


def run(state):
    entry = state["entry"]
    if entry == "block":
        A = S.SparseMatrix.from_csr(state["M"], state["K"], *state["csr"])
        return {"rowptr": A.bcsrRowPtr, "colidx": A.bcsrColIdx, "vals": A.bcsrVal}
    if entry == "call":
        S.spmm(state["A"], state["B"], state["C"])
    elif entry == "host":
        state["plan"].spmm_host(state["B"], state["C"])
    else:
        if entry == "update":
            state["plan"].set_values()
        state["plan"].spmm(state["B"], state["C"])
    return state["C"]


def _blocks_and_entries(case):
    """Expected numbers of stored blocks and of entries."""
    n, Mb, Kb, kind = case["M"], case["M"] // 16, case["K"] // 16, case["matrix"]
    if kind == "band":
        i, b = np.arange(Mb) * 16, case["half_bandwidth"]
        blocks = int((np.minimum(n - 1, i + 15 + b) // 16 - np.maximum(0, i - b) // 16 + 1).sum())
        return blocks, n * (2 * b + 1) - b * (b + 1)
    if kind == "layer":
        return case["fill"] * Mb * Kb, 256 * case["fill"] * Mb * Kb
    if kind == "uniform":
        return Mb * Kb * (1.0 - (1.0 - case["density"]) ** 256), case["density"] * n * n
    if kind == "powerlaw":  # per row, counted on matrices of this kind
        return n * (7.7 if case["order"] == "given" else 8.3), n * 14.0
    return n + 1, 0.3 * 256 * n


def work(case):
    """One pass: matrix, B and C (or CSR and blocks) moved once; two operations per stored value of a block and column."""
    M, K, N = case["M"], case["K"], case["N"]
    blocks, entries = _blocks_and_entries(case)
    matrix = 516 * blocks + 4 * (M // 16 + 1)
    if case["entry"] == "block":
        return {"bytes": 6 * entries + 4 * (M + 1) + matrix, "flops": 0}
    return {"bytes": matrix + 2 * N * K + 2 * M * N, "flops": 512 * blocks * N}


def tolerance(case):
    # Blocking moves values and indices.  A product has fp16 inputs, fp32 sums and one rounding to fp16 (2^-11 of the
    # value): another order of the sums moves a result by a unit in its last place now and then.
    return "exact" if case["entry"] == "block" else {"rel": 1e-3, "max": 4e-3}
