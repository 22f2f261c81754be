"""``torch.library`` registration of the SpMM, with a gradient for B, and a small CSR holder.

The reference's Python ops are plain pybind functions (torch_csrspmm/binding.cpp:26-32): opaque to
``torch.compile``, no ``out=``, no autograd, ``beta`` only ever multiplying a fresh zero tensor
(torch_csrspmm/torch_csrspmm_naive.cpp:32-34).  This module adds, on top of the same C ABI:

* ``torch.ops.csrspmm_b200.spmm(row_ptr, col_idx, values, B, alpha, kernel)`` -> new C, with a fake
  (meta) implementation so it traces, and an autograd formula for B:
  ``dB = alpha * A^T @ dC`` (A^T built once per matrix as a CSR, by a stable sort on the device);
* ``torch.ops.csrspmm_b200.spmm_(row_ptr, col_idx, values, B, C, alpha, beta, kernel)`` -> in place
  ``C = alpha * A @ B + beta * C`` (the reference's full semantics);
* ``CsrMatrix``: keeps the three arrays, the longest row (so AUTO can pick the row kernel), the cached
  transpose and, per dense width, the matrix's schedule (``csrspmm_b200_schedule_create``) together.

Gradients with respect to the stored values of A (a sampled dense-dense product) are not provided.
"""
from __future__ import annotations

import torch

from . import _lib, ops


def transpose_csr(row_ptr: torch.Tensor, col_idx: torch.Tensor, values: torch.Tensor, Kd: int):
    """CSR of A^T (Kd x M) from the CSR of A (M x Kd), on the arrays' device.  Entries of a column
    keep their row order (stable sort), so the result has ascending, distinct column indices
    whenever A has no repeated entry."""
    if (row_ptr.is_cuda and col_idx.is_cuda and values.is_cuda and row_ptr.dtype == col_idx.dtype == torch.int32
            and values.dtype == torch.float32 and not (values.requires_grad and torch.is_grad_enabled())
            and row_ptr.is_contiguous() and col_idx.is_contiguous() and values.is_contiguous() and Kd < 2**31 - 1):
        return _lib.binding().transpose(row_ptr, col_idx, values, int(Kd))
    # host arrays, other types and sizes
    M = row_ptr.numel() - 1
    lens = (row_ptr[1:] - row_ptr[:-1]).long()
    rows = torch.repeat_interleave(torch.arange(M, device=row_ptr.device, dtype=torch.int32), lens)
    order = torch.sort(col_idx.long(), stable=True).indices
    t_col = rows[order].contiguous()
    t_val = values[order].contiguous()
    counts = torch.bincount(col_idx.long(), minlength=Kd)
    t_rp = torch.zeros(Kd + 1, dtype=torch.int32, device=row_ptr.device)
    t_rp[1:] = torch.cumsum(counts, 0).to(torch.int32)
    return t_rp, t_col, t_val


# The operators' schemas and fake implementations; their CUDA kernels and the gradient are registered by the
# binding (csrc/torch/binding.cpp), which is loaded here when it has been built.
_library = torch.library.Library("csrspmm_b200", "DEF")
_library.define("spmm(Tensor row_ptr, Tensor col_idx, Tensor values, Tensor B, float alpha, str kernel) -> Tensor",
                tags=(torch.Tag.pt2_compliant_tag,))
_library.define("spmm_(Tensor row_ptr, Tensor col_idx, Tensor values, Tensor B, Tensor(a!) C, float alpha, float beta, "
                "str kernel) -> ()", tags=(torch.Tag.pt2_compliant_tag,))
_library.define("transpose(Tensor row_ptr, Tensor col_idx, Tensor values, SymInt Kd) -> (Tensor, Tensor, Tensor)",
                tags=(torch.Tag.pt2_compliant_tag,))


@torch.library.register_fake("csrspmm_b200::spmm")
def _spmm_fake(row_ptr, col_idx, values, B, alpha, kernel):
    return B.new_empty((row_ptr.shape[0] - 1, B.shape[1]))


@torch.library.register_fake("csrspmm_b200::spmm_")
def _spmm_inplace_fake(row_ptr, col_idx, values, B, C, alpha, beta, kernel):
    return None


@torch.library.register_fake("csrspmm_b200::transpose")
def _transpose_fake(row_ptr, col_idx, values, Kd):
    return row_ptr.new_empty((Kd + 1,)), torch.empty_like(col_idx), torch.empty_like(values)


try:
    _lib.binding()
except _lib.LibraryMissing:  # not built: the operators trace, and calling one on a GPU says there is no kernel
    pass

spmm_op = torch.ops.csrspmm_b200.spmm
spmm_inplace_op = torch.ops.csrspmm_b200.spmm_


class CsrMatrix:
    """A CSR matrix on a CUDA device together with what repeated products need: the longest row
    (lets AUTO choose the whole-row kernel when rows are even) and, on first use, the transpose."""

    def __init__(self, row_ptr: torch.Tensor, col_idx: torch.Tensor, values: torch.Tensor, shape, validate: bool = False):
        self.row_ptr, self.col_idx, self.values = row_ptr, col_idx, values
        self.shape = (int(shape[0]), int(shape[1]))
        if row_ptr.numel() != self.shape[0] + 1:
            raise ValueError("row_ptr must have shape[0] + 1 entries")
        if validate:
            ops.validate_csr(row_ptr, col_idx, self.shape[1])
        self.max_row_nnz = ops.row_stats(row_ptr)["max_row_nnz"] if row_ptr.is_cuda else 0
        self._t = None
        self._schedules = {}  # dense width -> ops.Schedule or None (built on first use, kept with the matrix)

    def schedule(self, Nd: int):
        """The per-matrix schedule for a B of ``Nd`` columns, built on first use (a few milliseconds) and kept;
        None when the library finds nothing worth scheduling for this matrix and width."""
        if Nd not in self._schedules:
            Nd = int(Nd)
            sched = None
            if self.row_ptr.is_cuda and self.nnz > 0:
                sched = ops.Schedule(self.row_ptr, self.col_idx, self.shape[1], Nd)
                if not sched.active:
                    sched.close()
                    sched = None
            self._schedules[Nd] = sched
        return self._schedules[Nd]

    @property
    def nnz(self) -> int:
        return int(self.col_idx.numel())

    def t(self) -> "CsrMatrix":
        if self._t is None:
            rp, ci, va = transpose_csr(self.row_ptr, self.col_idx, self.values, self.shape[1])
            self._t = CsrMatrix(rp, ci, va, (self.shape[1], self.shape[0]))
            self._t._t = self
        return self._t

    def matmul(self, B: torch.Tensor, alpha: float = 1.0, *, out: torch.Tensor | None = None, beta: float = 0.0,
               kernel: str = "auto") -> torch.Tensor:
        """alpha * A @ B (+ beta * out).  Differentiable in B when ``out`` is None."""
        sched = self.schedule(B.shape[1]) if kernel == "auto" else None
        if out is None and B.requires_grad:
            return _lib.binding().matmul(self, self.row_ptr, self.col_idx, self.values, B, alpha, _lib.KERNEL_IDS[kernel],
                                         self.max_row_nnz, sched.handle if sched is not None else 0)
        return ops.spmm(self.row_ptr, self.col_idx, self.values, B, out, alpha, beta, kernel=kernel,
                        max_row_nnz=self.max_row_nnz, schedule=sched)

    def _transpose_parts(self, Nd: int, kernel: int):
        """What the backward product of ``matmul`` needs (called from the binding)."""
        At = self.t()
        sched = At.schedule(Nd) if kernel == _lib.KERNEL_AUTO else None
        return At.row_ptr, At.col_idx, At.values, At.max_row_nnz, sched.handle if sched is not None else 0

    __matmul__ = matmul
