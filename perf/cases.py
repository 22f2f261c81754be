"""Timing cases of the library: the calls its users make, over the sizes they make them at.

Every case names one family, i.e. one public entry point and the state a program keeps for it:

    op       one of the five drop-in ops of ``torch_csrspmm``: arrays and B in, a new C out
    update   ``ops.spmm`` into an existing C with beta (iterative methods, accumulating layers)
    loop     ``ops.SpmmCall``, a product prepared once and repeated
    graph    ``CsrMatrix @ B``: aggregation over a fixed graph (inference)
    train    ``CsrMatrix @ B`` and the gradient of B (training on a fixed graph)
    sampled  ``torch.ops.csrspmm_b200.spmm`` and the gradient of B: the matrix is new at each step (a
             sampled subgraph), so the backward product transposes it every time
    e2m1     ``ops.spmm`` with packed 4-bit values
    compress a dense weight to CSR (``ops.dense2csr``) and its values to 4 bits (``ops.e2m1_quantize``)
    host     ``ops.spmm_host``: operands and result in pinned host memory

Matrices have columns uniform in each row, ascending, and row lengths that are either even (each
entry present independently) or Zipf-distributed (rescaled to the mean, capped), as in
``csrspmm_b200.generators``; repeats that a row draws are dropped.
"""
import math

import numpy as np
import torch

import torch_csrspmm
from csrspmm_b200 import ops
from csrspmm_b200.torch_library import CsrMatrix

OPS = ("naive", "warp_per_row", "warp_per_row_smem", "warp_per_row_fp4", "warp_per_row_smem_fp4")


def _case(family, M, Kd, Nd, mean, zipf=0.0, cap=0, **more):
    return dict(family=family, M=M, Kd=Kd, Nd=Nd, mean=float(mean), zipf=float(zipf), cap=cap, **more)


def listed():
    return [
        # the smallest call: the 1024 x 1024 check problem through a drop-in op
        dict(_case("op", 1024, 1024, 64, 10.24, op="warp_per_row_fp4", alpha=1.0), name="op_check"),
        # the largest shape of the torch op table (a pruned layer: few columns, a wide B), one density of its range
        dict(_case("op", 8192, 256, 4096, 25.6, op="warp_per_row_smem_fp4", alpha=1.1), name="op_wide"),
        # the "large" shape of the kernel sweep: C = A B + 0.5 C in place
        dict(_case("update", 4096, 4096, 128, 409.6, alpha=1.0, beta=0.5), name="update_large"),
        # the medium uniform configuration in a tight loop
        dict(_case("loop", 16384, 16384, 128, 16.384, alpha=1.0), name="loop_medium"),
        # power-law graph aggregation
        dict(_case("graph", 1 << 20, 1 << 20, 64, 16, zipf=2.0, cap=16384), name="graph_powerlaw"),
        # nothing a multiple of anything: rectangular graph block, 50 features
        dict(_case("graph", 100003, 77777, 50, 11, zipf=2.1, cap=4999), name="graph_ragged"),
        # a wide product of the largest kind: hub rows, 2 KB rows of B, B many times L2
        dict(_case("graph", 1 << 22, 1 << 22, 512, 32, zipf=2.2, cap=65536), name="graph_xl"),
        # forward and backward on a fixed graph of a quarter of the power-law configuration's rows
        dict(_case("train", 1 << 18, 1 << 18, 128, 16, zipf=2.0, cap=16384), name="train_graph"),
        # forward and backward on a subgraph that is new each step
        dict(_case("sampled", 65536, 65536, 64, 16), name="train_sampled"),
        # long even rows with packed 4-bit values
        dict(_case("e2m1", 65536, 65536, 256, 327.68, alpha=1.0), name="e2m1_long_rows"),
        # a pruned 4096 x 4096 weight compressed on the device
        dict(_case("compress", 4096, 4096, 0, 409.6), name="compress_weight"),
        # a product that starts and ends in host memory
        dict(_case("host", 1 << 18, 1 << 18, 64, 16, zipf=2.0, cap=16384), name="host_round_trip"),
    ]


# The ranges, log-uniform: rows, columns of A, columns of B, mean row.  draw() rejects what has more than 4e7
# entries, 1e10 multiply-adds or 5e8 dense elements (host, compress: 1.2e8).  "layer" is the op family on the shapes of the
# torch op table: few columns of A, a wide B.
RANGES = {
    "op": ((512, 65536), (64, 65536), (16, 4096), (2, 512)),
    "layer": ((512, 16384), (64, 1024), (512, 4096), (2, 300)),
    "update": ((512, 65536), (1024, 65536), (16, 512), (2, 1024)),
    "loop": ((1024, 262144), (1024, 262144), (16, 512), (2, 512)),
    "graph": ((2048, 1 << 21), (2048, 1 << 21), (1, 512), (2, 48)),
    "train": ((2048, 1 << 19), (2048, 1 << 19), (8, 512), (2, 48)),
    "sampled": ((512, 1 << 18), (512, 1 << 18), (8, 512), (2, 48)),
    "e2m1": ((1024, 131072), (1024, 131072), (16, 1024), (8, 512)),
    "compress": ((256, 16384), (256, 16384), (0, 0), (2, 2048)),
    "host": ((4096, 1 << 19), (4096, 1 << 19), (16, 512), (2, 48)),
}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(sorted(set(RANGES) - {"layer"}))
    rows, cols, width, mean = RANGES["layer" if family == "op" and rng.random() < 0.5 else family]
    while True:
        M, Kd = _log(rng, *rows), _log(rng, *cols)
        if rng.random() < 0.4:  # square, as graphs are
            Kd = M
        Nd = 0
        if family != "compress":
            Nd = _log(rng, *width)
            if rng.random() < 0.75 and Nd >= 8:  # most widths are whole vectors
                step = 4 if Nd < 64 else 32
                Nd = max(step, (Nd + step // 2) // step * step)
        m = math.exp(rng.uniform(math.log(mean[0]), math.log(mean[1])))
        m = round(min(m, 0.3 * Kd), 3)
        nnz, dense = M * m, float(M + Kd) * max(Nd, 1)
        if family == "compress":
            dense = float(M) * Kd
        if m < 1 or nnz > 4e7 or nnz * Nd > 1e10 or dense > (1.2e8 if family in ("host", "compress") else 5e8):
            continue
        break
    uneven = family in ("graph", "train", "host") and rng.random() < 0.7 or family in ("update", "sampled", "loop") and rng.random() < 0.25
    zipf, cap = 0.0, 0
    if uneven:
        zipf = round(rng.uniform(1.9, 2.4), 2)
        cap = max(4, min(65536, Kd // 64, int(m * 1024)))
        uneven = cap > 4 * m
    case = _case(family, M, Kd, Nd, m, zipf if uneven else 0.0, cap if uneven else 0)
    if family in ("op", "update", "loop", "e2m1"):
        case["alpha"] = rng.choice([1.0, 1.1])
    if family == "op":
        case["op"] = rng.choice(OPS)
    if family == "update":
        case["beta"] = rng.choice([0.5, 1.0])
    return case


# ---- inputs -----------------------------------------------------------------------------------------

def _lengths(case, seed, gen):
    """Entries per row before repeats are dropped (int64 on the GPU)."""
    M, Kd, mean = case["M"], case["Kd"], case["mean"]
    if not case["zipf"]:
        p = torch.full((M,), mean / Kd, device="cuda")
        return torch.binomial(torch.full((M,), float(Kd), device="cuda"), p, generator=gen).long()
    z = torch.from_numpy(np.random.default_rng(seed).zipf(case["zipf"], size=M)).cuda().double()
    lo, hi = 1e-6, 2.0 * mean
    for _ in range(40):  # the factor that gives the mean after rounding and clipping
        mid = 0.5 * (lo + hi)
        if float((z * mid).round_().clamp_(1, case["cap"]).mean()) < mean:
            lo = mid
        else:
            hi = mid
    return (z * hi).round_().clamp_(1, case["cap"]).long()


def _csr(case, seed, gen):
    """(row_ptr, col_idx, values) on the GPU."""
    M, Kd = case["M"], case["Kd"]
    if case["mean"] > 0.02 * Kd and M * Kd <= 1 << 28 and not case["zipf"]:  # dense enough for a mask
        at = (torch.rand((M, Kd), generator=gen, device="cuda") < case["mean"] / Kd).nonzero()
        rows, cols = at[:, 0], at[:, 1].to(torch.int32)
    else:
        lens = _lengths(case, seed, gen)
        rows = torch.repeat_interleave(torch.arange(M, device="cuda"), lens)
        key = rows * Kd + torch.randint(0, Kd, rows.shape, generator=gen, device="cuda")
        key = torch.unique_consecutive(key.sort().values)
        rows = torch.div(key, Kd, rounding_mode="floor")
        cols = (key - rows * Kd).to(torch.int32)
    row_ptr = torch.zeros(M + 1, dtype=torch.int32, device="cuda")
    row_ptr[1:] = torch.bincount(rows, minlength=M).cumsum(0)
    values = torch.empty(cols.shape, device="cuda").uniform_(-1.0, 1.0, generator=gen)
    return row_ptr, cols.contiguous(), values


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    family, M, Kd, Nd = case["family"], case["M"], case["Kd"], case["Nd"]
    if family == "compress":
        dense = torch.zeros(M * Kd, device="cuda")
        at = torch.randperm(M * Kd, generator=gen, device="cuda")[: round(M * case["mean"])]
        dense[at] = torch.randn(at.shape, generator=gen, device="cuda")
        return dict(case=case, dense=dense.view(M, Kd))
    rp, ci, va = _csr(case, int(seed), gen)
    B = torch.randn((Kd, Nd), generator=gen, device="cuda")
    s = dict(case=case, rp=rp, ci=ci, va=va, B=B)
    if family == "op":
        s["longest"] = int((rp[1:] - rp[:-1]).max())
    elif family == "update":
        s["C"] = torch.randn((M, Nd), generator=gen, device="cuda")
        s["longest"] = ops.row_stats(rp)["max_row_nnz"]
    elif family == "loop":
        longest = ops.row_stats(rp)["max_row_nnz"]
        s["call"] = ops.SpmmCall(rp, ci, va, B, torch.empty((M, Nd), device="cuda"), case["alpha"], 0.0, max_row_nnz=longest)
    elif family == "graph":
        s["A"] = CsrMatrix(rp, ci, va, (M, Kd))
    elif family == "train":
        s["A"] = CsrMatrix(rp, ci, va, (M, Kd))
        B.requires_grad_(True)
        s["G"] = torch.randn((M, Nd), generator=gen, device="cuda")
    elif family == "sampled":
        B.requires_grad_(True)
        s["G"] = torch.randn((M, Nd), generator=gen, device="cuda")
    elif family == "e2m1":
        s["longest"] = ops.row_stats(rp)["max_row_nnz"]
        s["nnz"] = int(va.numel())
        s["packed"], s["scale"] = ops.e2m1_quantize(va)
        del s["va"]
    elif family == "host":
        for k in ("rp", "ci", "va", "B"):
            s[k] = s[k].cpu().pin_memory()
        s["C"] = torch.empty((M, Nd), pin_memory=True)
    return s


# ---- one pass ---------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    family = case["family"]
    if family == "op":
        op = getattr(torch_csrspmm, "csrspmm_" + case["op"])
        if "smem" in case["op"]:  # these two take the longest row as well
            return op(s["rp"], s["ci"], s["va"], s["longest"], s["B"], case["alpha"], 0.0)
        return op(s["rp"], s["ci"], s["va"], s["B"], case["alpha"], 0.0)
    if family == "update":
        return ops.spmm(s["rp"], s["ci"], s["va"], s["B"], s["C"], case["alpha"], case["beta"], max_row_nnz=s["longest"])
    if family == "loop":
        return s["call"]()
    if family == "graph":
        return s["A"] @ s["B"]
    if family in ("train", "sampled"):
        out = s["A"] @ s["B"] if family == "train" else torch.ops.csrspmm_b200.spmm(s["rp"], s["ci"], s["va"], s["B"], 1.0, "auto")
        (dB,) = torch.autograd.grad(out, s["B"], s["G"])
        return {"out": out.detach(), "dB": dB}
    if family == "e2m1":
        return ops.spmm(s["rp"], s["ci"], s["packed"], s["B"], None, case["alpha"], 0.0, e2m1_scale=s["scale"],
                        nnz=s["nnz"], max_row_nnz=s["longest"])
    if family == "compress":
        rp, ci, va, longest = ops.dense2csr(s["dense"])
        packed, scale = ops.e2m1_quantize(va)
        return {"row_ptr": rp, "col_idx": ci, "values": va, "longest": longest, "packed": packed, "scale": scale}
    return ops.spmm_host(s["rp"], s["ci"], s["va"], s["B"], s["C"])


def work(case):
    """Each operand once: the stored entries, the row offsets, the rows of B that are named, C."""
    family, M, Kd, Nd = case["family"], case["M"], case["Kd"], case["Nd"]
    nnz = M * case["mean"]
    if family == "compress":
        return {"bytes": 4.0 * M * Kd + 8.5 * nnz + 4.0 * (M + 1), "flops": 0.0}
    touched = Kd * (1.0 - math.exp(-nnz / Kd))
    matrix = nnz * (4.5 if family == "e2m1" else 8.0) + 4.0 * (M + 1)
    n_bytes = matrix + 4.0 * Nd * (touched + M * (2 if case.get("beta") else 1))
    flops = 2.0 * nnz * Nd
    if family in ("train", "sampled"):  # dB = A^T G: the matrix and G in, dB out
        n_bytes += matrix + 4.0 * Nd * (M + Kd)
        flops *= 2
    return {"bytes": n_bytes, "flops": flops}


def tolerance(case):
    """fp32 sums in another order differ by some 1e-6 of the result; a conversion has one right answer."""
    return "exact" if case["family"] == "compress" else {"rel": 1e-5}
