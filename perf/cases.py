"""The workloads whose speed is measured, as calls a user's program makes.

The operators are those of the hybrid sparse path: building the format from a CSR matrix, multiplying
with it (inference, training, a GCN layer stack), sampled dense-dense products over its pattern, and the
host-buffer calls of the reference's extension modules.  Matrices are the seeded graphs of the
benchmark configurations (uniform, clustered, R-MAT) and sizes around them; feature widths are hidden sizes
(multiples of 32), other multiples of 8, and class counts, which may be any number.

A state holds what a program keeps between calls: the CSR arrays, the built format with its plan, weights
and input features.
"""
from __future__ import annotations

import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "tr-spmm_zzx_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import Libra5BlockOnline  # noqa: E402
import Libra6SpMMOnline  # noqa: E402
import trspmm  # noqa: E402
from trspmm import graphs  # noqa: E402


def _uniform(n, per_row):
    return {"graph": "uniform", "n": n, "per_row": per_row}


def _clustered(n, community=128, intra=24, glob=4):
    return {"graph": "clustered", "n": n, "community": community, "intra": intra, "glob": glob}


def _rmat(scale, ef):
    return {"graph": "rmat", "scale": scale, "ef": ef}


def listed():
    return [
        # one small layer of a small graph: what a call costs before any work is done
        {"name": "spmm uniform 4k F64", "op": "spmm", **_uniform(4096, 16), "F": 64, "out": "f16", "strict": False},
        # a community graph whose windows share columns: the case the dense blocks exist for
        {"name": "spmm clustered 262k F128", "op": "spmm", **_clustered(262144), "F": 128, "out": "f16", "strict": False},
        # the headline benchmark: a power-law graph with hub windows, inputs far beyond the L2
        {"name": "spmm rmat21 F128", "op": "spmm", **_rmat(21, 32), "F": 128, "out": "f16", "strict": False},
        # an output layer: the width is a class count, nothing is a multiple of 8, fp32 logits, lossless format
        {"name": "spmm rmat17 F47 f32", "op": "spmm", **_rmat(17, 16), "F": 47, "out": "f32", "strict": True},
        # attention-like scores on a pattern planned once
        {"name": "sddmm plan clustered 262k K64", "op": "sddmm_plan", **_clustered(262144), "K": 64},
        # the same product on a pattern that is used once, ragged rows, a width that is no power of two
        {"name": "sddmm uniform 50021 K96", "op": "sddmm", **_uniform(50021, 16), "K": 96},
        # one training step of a layer: forward, gradient of the features and of the edge weights
        {"name": "train rmat18 F64", "op": "train", **_rmat(18, 16), "F": 64},
        # two-layer GCN inference
        {"name": "gcn rmat20 256-128-64", "op": "gcn", **_rmat(20, 16), "F0": 256, "F1": 128, "F2": 64},
        # a new matrix arrives on the device and is put into the format
        {"name": "build clustered 262k", "op": "build", **_clustered(262144), "density": 8, "strict": False},
        # the reference's builder module: CPU tensors in, CPU arrays out
        {"name": "module build rmat15", "op": "module_build", **_rmat(15, 16), "density": 8},
        # the reference's SpMM module: every array a CPU tensor, everything inside the one call
        {"name": "module spmm clustered 65k F128", "op": "module_spmm", **_clustered(65536), "F": 128, "epoches": 1},
        # the matrix stays on the GPU, features come from and results go back to pinned host memory
        {"name": "resident rmat18 F128", "op": "resident", **_rmat(18, 16), "F": 128, "out": "f16"},
    ]


# Largest number of nodes drawn per operator: bounded by the listed case of the operator that costs most.
_MAX_NODES = {"spmm": 1 << 20, "sddmm_plan": 1 << 19, "sddmm": 1 << 18, "train": 1 << 18, "gcn": 1 << 20,
              "build": 1 << 18, "module_build": 1 << 15, "module_spmm": 1 << 16, "resident": 1 << 18}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng):
    """Hidden sizes, other multiples of 8, class counts."""
    kind = rng.random()
    if kind < 0.5:
        return rng.choice((32, 64, 128, 256))
    if kind < 0.75:
        return 8 * _log_int(rng, 2, 32)
    return _log_int(rng, 7, 256)


def draw(rng):
    ops = ("spmm", "spmm", "spmm", "spmm", "sddmm_plan", "sddmm", "train", "gcn", "build", "module_build",
           "module_spmm", "resident")
    op = rng.choice(ops)
    nodes = _log_int(rng, 2048, _MAX_NODES[op])
    kind = rng.choice(("uniform", "clustered", "rmat"))
    if kind == "uniform":
        g = _uniform(nodes, rng.randint(4, 32))
    elif kind == "clustered":
        g = _clustered(nodes, rng.choice((64, 128, 256)), rng.randint(12, 32), rng.randint(1, 6))
    else:
        g = _rmat(max(11, int(math.log2(nodes))), rng.choice((8, 16, 24)))
    case = {"op": op, **g}
    if op == "spmm":
        case.update(F=_width(rng), out=rng.choice(("f16", "f16", "f32")), strict=rng.random() < 0.25)
    elif op in ("sddmm_plan", "sddmm"):
        case.update(K=_width(rng))
    elif op == "train":
        case.update(F=_width(rng))
    elif op == "gcn":
        case.update(F0=rng.choice((64, 128, 256)), F1=rng.choice((32, 64, 128)), F2=_log_int(rng, 7, 64))
    elif op == "build":
        case.update(density=rng.choice((4, 8)), strict=rng.random() < 0.5)
    elif op == "module_build":
        case.update(density=rng.choice((4, 8)))
    elif op == "module_spmm":
        case.update(F=rng.choice((32, 64, 128)), epoches=rng.choice((1, 5)))
    else:
        case.update(F=_width(rng), out=rng.choice(("f16", "f32")))
    return case


def _roll_windows(rowptr, col, val, shift, window=16):
    """The same matrix with its full 16-row windows rotated by `shift` (a ragged last window stays last)."""
    n = rowptr.numel() - 1
    full = n // window * window
    rows = torch.arange(n, device=rowptr.device)
    rows[:full] = torch.roll(rows[:full], (shift % max(full // window, 1)) * window)
    deg = (rowptr[1:] - rowptr[:-1]).long()[rows]
    out = torch.zeros(n + 1, dtype=torch.int64, device=rowptr.device)
    out[1:] = torch.cumsum(deg, 0)
    src = torch.repeat_interleave(rowptr[:-1].long()[rows] - out[:-1], deg) + torch.arange(col.numel(), device=col.device)
    return out.to(torch.int32), col[src], val[src]


# Operators with one result per entry (or arrays sized by the pattern).  Their matrices come from one graph per case and
# differ between seeds in where the windows lie and in the values, so that the lengths of the results are the same.
_PER_ENTRY = ("sddmm", "sddmm_plan", "train", "build", "module_build")


def _csr(case, seed):
    if case["op"] in _PER_ENTRY:
        rowptr, col, val = _roll_windows(*_graph(case, 0), shift=1 + seed)
        return rowptr, col, val * (1.0 + _randn(val.shape, seed + 7, 0.1).float())
    return _graph(case, seed)


def _graph(case, seed):
    if case["graph"] == "uniform":
        return graphs.uniform_graph(case["n"], case["per_row"], seed=seed, device="cuda")
    if case["graph"] == "clustered":
        return graphs.clustered_graph(case["n"], case["community"], case["intra"], case["glob"], seed=seed, device="cuda")
    return graphs.rmat_graph(case["scale"], case["ef"], seed=seed, device="cuda")


def _randn(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * scale).half()


_OUT = {"f16": torch.float16, "f32": torch.float32}


def prepare(case, seed):
    op = case["op"]
    rowptr, col, val = _csr(case, seed)
    n = rowptr.numel() - 1
    s = {"op": op, "n": n}
    if op == "spmm":
        fmt, _ = trspmm.build_format(rowptr, col, val, strict=case["strict"])
        s.update(plan=trspmm.SpmmPlan(fmt, n, n), B=_randn((n, case["F"]), seed + 1), out=_OUT[case["out"]])
    elif op == "sddmm_plan":
        s.update(plan=trspmm.SddmmPlan(rowptr, col, n), X=_randn((n, case["K"]), seed + 1), Y=_randn((n, case["K"]), seed + 2))
    elif op == "sddmm":
        s.update(rowptr=rowptr, col=col, X=_randn((n, case["K"]), seed + 1), Y=_randn((n, case["K"]), seed + 2))
    elif op == "train":
        s.update(layer=trspmm.DifferentiableSpmm(rowptr, col, val, n), values=val.clone().requires_grad_(),
                 B=_randn((n, case["F"]), seed + 1).requires_grad_(), dC=_randn((n, case["F"]), seed + 2))
    elif op == "gcn":
        s.update(gcn=trspmm.ShardedGCN2(rowptr, col, val), X=_randn((n, case["F0"]), seed + 1),
                 W1=_randn((case["F0"], case["F1"]), seed + 2, 0.02), W2=_randn((case["F1"], case["F2"]), seed + 3, 0.02))
    elif op == "build":
        s.update(rowptr=rowptr, col=col, val=val, density=case["density"], strict=case["strict"])
    elif op == "module_build":
        s.update(rowptr=rowptr.cpu(), col=col.cpu(), val=val.cpu(), density=case["density"])
    elif op == "module_spmm":
        fmt, _ = trspmm.build_format(rowptr, col, val)
        s.update(fmt=fmt.half_values().to("cpu"), B=_randn((n, case["F"]), seed + 1).cpu(), F=case["F"], epoches=case["epoches"])
    else:
        fmt, _ = trspmm.build_format(rowptr, col, val)
        s.update(op_=trspmm.ResidentSpmm(fmt, n, n, max_dimN=case["F"]), B=_randn((n, case["F"]), seed + 1).cpu().pin_memory(),
                 C=torch.empty((n, case["F"]), dtype=_OUT[case["out"]]).pin_memory())
    return s


def run(s):
    op = s["op"]
    if op == "spmm":
        return s["plan"].run(s["B"], out_dtype=s["out"])
    if op == "sddmm_plan":
        return s["plan"].run(s["X"], s["Y"])
    if op == "sddmm":
        return trspmm.sddmm(s["rowptr"], s["col"], s["X"], s["Y"])
    if op == "train":
        C = s["layer"](s["B"], values=s["values"])
        return (C, *torch.autograd.grad(C, (s["B"], s["values"]), s["dC"]))
    if op == "gcn":
        return s["gcn"].forward(s["X"], s["W1"], s["W2"])
    if op == "build":
        fmt, _ = trspmm.build_format(s["rowptr"], s["col"], s["val"], density=s["density"], strict=s["strict"])
        return fmt.arrays()
    if op == "module_build":  # partSize_t, partSize_c, shortSize, density, window, wide, tc_min_util, sptc_min_util, sptc_threshold
        return Libra5BlockOnline.block_sptc_2to4_online(s["rowptr"], s["col"], s["val"], 32, 32, 3, s["density"], 16, 16,
                                                        0.0, 0.5, 12)[:-1]  # the last one is the build time
    if op == "module_spmm":
        f, n = s["fmt"], s["n"]
        return Libra6SpMMOnline.forward_fp16_tcu_cuda_sptc_mma_parallel_online(
            f.t_row_offset, f.t_block_offset, f.t_column, f.t_value, f.t_window_row, f.t_atomic, f.t_binary,
            f.c_row_offset, f.c_row, f.c_atomic, f.c_column, f.c_value,
            f.cs_row_offset, f.cs_row, f.cs_atomic, f.cs_column, f.cs_value,
            f.s_column, f.s_value, f.s_pos, f.s_offset, f.s_tile_window, f.s_tile_column, f.s_packed_a, f.s_packed_meta,
            f.s_window_tile_offset, s["B"],
            f.t_atomic.numel(), f.c_atomic.numel(), 32, f.cs_atomic.numel(), 16, s["F"], n, n, s["epoches"])[0]
    return s["op_"].forward(s["B"], s["C"])[0]


def _counts(case):
    """Expected (rows, entries, distinct (16-row window, column) pairs) of the case's graph."""
    if case["graph"] == "uniform":
        n, k = case["n"], case["per_row"]
        return n, n * (k + 1), n * (k + 1)
    if case["graph"] == "clustered":
        n, m = case["n"], min(case["community"], case["n"])
        intra = m * (1.0 - (1.0 - 1.0 / m) ** (2 * case["intra"]))
        glob = 2.0 * case["glob"] + 1.0
        pairs = m * (1.0 - (1.0 - intra / m) ** 16) / 16.0
        return n, int(n * (intra + glob)), int(n * (pairs + glob))
    # R-MAT: the expected number of distinct cells, cells grouped by how often each quadrant was taken
    scale, m = case["scale"], 2.0 * case["ef"] * (1 << case["scale"])
    nnz = float(1 << scale)
    for i in range(scale + 1):
        for j in range(scale + 1 - i):
            k = scale - i - j
            cells = math.comb(scale, i) * math.comb(scale - i, j) * 2.0 ** k
            nnz += cells * -math.expm1(-m * 0.57 ** i * 0.05 ** j * 0.19 ** k)
    return 1 << scale, int(nnz), int(0.85 * nnz)


def work(case):
    """Bytes: entries as 4-byte column + 2-byte value, row pointers, every dense operand once.  Flops: 2 per entry and
    feature, and the dense products of the GCN."""
    op = case["op"]
    n, nnz, pairs = _counts(case)
    csr = 6 * nnz + 4 * (n + 1)
    if op in ("spmm", "module_spmm", "resident"):
        F = case["F"]
        out = 2 if case.get("out") == "f16" else 4
        return {"bytes": csr + 2 * n * F + out * n * F, "flops": 2 * nnz * F * case.get("epoches", 1)}
    if op in ("sddmm", "sddmm_plan"):
        return {"bytes": csr + 4 * n * case["K"], "flops": 2 * nnz * case["K"]}
    if op == "train":  # forward and transposed product over one pattern each, the sampled product: B and dC in, C and dB out
        F = case["F"]
        return {"bytes": 2 * csr + 4 * nnz + 8 * n * F, "flops": 6 * nnz * F}
    if op == "gcn":
        f0, f1, f2 = case["F0"], case["F1"], case["F2"]
        return {"bytes": 2 * csr + 2 * n * (f0 + f2), "flops": 2 * n * f1 * (f0 + f2) + 2 * nnz * (f1 + f2)}
    # builder: CSR in; per group of four columns 196 bytes of un-packed arrays and a quarter of a 360-byte packed tile out
    return {"bytes": 8 * nnz + 4 * n + int(71.5 * pairs), "flops": 0}


def tolerance(case):
    op = case["op"]
    if op in ("build", "module_build"):
        return "exact"
    if op == "gcn":
        return {"rel": 2e-3}  # two layers with fp16 activations between them
    if op == "module_spmm" or case.get("out") == "f32":
        return {"rel": 2e-5}  # fp32 sums of fp16 products in another order
    return {"rel": 1e-3}      # fp16 results
