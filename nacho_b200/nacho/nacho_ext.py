"""Host-side mirror of the reference's generated extension module ``nacho_ext``: the GPU tensor
classes and the ``gpu_<kernel>_f32`` operators, with the names, argument order, defaults and
read-only attributes the reference's binding generator emits
(src/backend/generate_bindings.cpp:84-154 classes, :288-331 operators, :317-327 keyword names
and the 256 x 256 default grid). Every operator forwards to the C ABI in ``libnacho_b200.so``
through the compiled module ``_native``; nothing is computed in Python or torch.

Tensors are 1-D contiguous CUDA torch tensors (int32 indices, float32 values) and ``shape`` is
a host int32 tensor, as in runtime/nacho_nb.h:22-31. Operands are borrowed; results are fresh
torch tensors owned by the returned object.
"""
from __future__ import annotations

import ctypes as C

import torch

from .. import _capi
from .._capi import Coo3Struct, CsrStruct, Csf3Struct

try:
    from .. import _native
except ImportError as e:
    raise ImportError("nacho_b200/_native.so is missing or does not load: build it with `python -m nacho_b200.build`. "
                      "nacho_b200 has no fallback path.") from e

__all__ = ["CSR_gpu", "COO3_gpu", "CSF3_gpu", "COO_gpu", "DCSR_gpu", "Scalar_gpu", "gpu_csr_add_f32", "gpu_csr_add_3_f32",
           "gpu_csr_mul_f32", "gpu_spgemm_f32", "gpu_coo3d_add_f32", "gpu_csf_add_f32", "gpu_coo_add_f32", "gpu_coo_mul_f32",
           "gpu_coo_csr_add_f32", "gpu_dcsr_add_f32", "gpu_dcsr_mul_f32", "gpu_dcsr_mul_without_recursive_partitioning_f32",
           "gpu_inner_prod_f32", "gpu_inner_prod_coo_f32", "gpu_sssmm_f32"]


def _dev_array(t, dtype, name):
    if not isinstance(t, torch.Tensor):
        raise TypeError(f"{name}: expected a torch tensor")
    if not t.is_cuda or t.dtype != dtype or t.dim() != 1 or not t.is_contiguous():
        raise TypeError(f"{name}: expected a 1-D contiguous CUDA tensor of dtype {dtype}")
    return t


def _shape_array(t, rank, name="shape"):
    if not isinstance(t, torch.Tensor):
        t = torch.tensor(list(t), dtype=torch.int32)
    if t.is_cuda or t.dtype != torch.int32 or t.dim() != 1 or t.numel() != rank:
        raise TypeError(f"{name}: expected a host int32 tensor of {rank} entries")
    return t.contiguous()


def _dims(shape):
    return tuple(shape.tolist())


def _host_shape(t):
    """``shape`` of a tensor object: the caller's host tensor, or for an operator's result one made when asked for."""
    try:
        return t._shape
    except AttributeError:
        t._shape = torch.tensor(t._dims, dtype=torch.int32)
        return t._shape


class CSR_gpu:
    """CSR matrix on the GPU: ``CSR_gpu(dim_j_offsets, dim_j_indices, values, shape)``
    (attribute names as emitted by src/backend/generate_bindings.cpp:84-154)."""

    __slots__ = ("_offsets", "_indices", "_values", "_shape", "_dims")

    def __init__(self, dim_j_offsets, dim_j_indices, values, shape):
        self._offsets = _dev_array(dim_j_offsets, torch.int32, "dim_j_offsets")
        self._indices = _dev_array(dim_j_indices, torch.int32, "dim_j_indices")
        self._values = _dev_array(values, torch.float32, "values")
        self._shape = _shape_array(shape, 2)
        self._dims = _dims(self._shape)
        if self._indices.numel() != self._values.numel():
            raise ValueError("dim_j_indices and values differ in length")
        if self._offsets.numel() != self._dims[0] + 1:
            raise ValueError("dim_j_offsets must hold rows + 1 entries")
        if not (self._offsets.device == self._indices.device == self._values.device):
            raise ValueError("all buffers of a tensor must live on one device")

    dim_j_offsets = property(lambda self: self._offsets)
    dim_j_indices = property(lambda self: self._indices)
    values = property(lambda self: self._values)
    shape = property(_host_shape)

    @property
    def device(self):
        return self._values.device

    def _struct(self) -> CsrStruct:
        return CsrStruct(*self._dims, self._values.numel(),
                         self._offsets.data_ptr(), self._indices.data_ptr(), self._values.data_ptr())

    def __repr__(self):
        return f"CSR_gpu(shape={self._dims}, nnz={self._values.numel()})"


def gpu_csr_add_f32(a: CSR_gpu, b: CSR_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> CSR_gpu:
    """Z = A + B (sorted union per row; explicit zeros kept). ``num_blocks`` and
    ``threads_per_block`` are accepted for compatibility and ignored."""
    return _native.csr_add(a, b)


def gpu_csr_mul_f32(a: CSR_gpu, b: CSR_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> CSR_gpu:
    """Z = A .* B (sorted intersection per row)."""
    return _native.csr_mul(a, b)


def gpu_csr_add_3_f32(a: CSR_gpu, b: CSR_gpu, c: CSR_gpu, num_blocks: int = 256,
                      threads_per_block: int = 256) -> CSR_gpu:
    """Z = (A + B) + C, the reference's association."""
    return _native.csr_add_3(a, b, c)


def gpu_spgemm_f32(a: CSR_gpu, b: CSR_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> CSR_gpu:
    """C = A @ B by expand-sort-compress; sorted columns per row, explicit zeros kept."""
    return _native.spgemm(a, b)


class COO3_gpu:
    """3-mode tensor as parallel coordinate arrays:
    ``COO3_gpu(dim_i_indices, dim_j_indices, dim_k_indices, values, shape)``."""

    __slots__ = ("_i", "_j", "_k", "_values", "_shape", "_dims")

    def __init__(self, dim_i_indices, dim_j_indices, dim_k_indices, values, shape):
        self._i = _dev_array(dim_i_indices, torch.int32, "dim_i_indices")
        self._j = _dev_array(dim_j_indices, torch.int32, "dim_j_indices")
        self._k = _dev_array(dim_k_indices, torch.int32, "dim_k_indices")
        self._values = _dev_array(values, torch.float32, "values")
        self._shape = _shape_array(shape, 3)
        self._dims = _dims(self._shape)
        n = self._values.numel()
        if not (self._i.numel() == self._j.numel() == self._k.numel() == n):
            raise ValueError("coordinate arrays and values differ in length")

    dim_i_indices = property(lambda self: self._i)
    dim_j_indices = property(lambda self: self._j)
    dim_k_indices = property(lambda self: self._k)
    values = property(lambda self: self._values)
    shape = property(_host_shape)

    @property
    def device(self):
        return self._values.device

    def _struct(self) -> Coo3Struct:
        dims = (C.c_int32 * 3)(*self._dims)
        return Coo3Struct(dims, self._values.numel(), self._i.data_ptr(), self._j.data_ptr(), self._k.data_ptr(),
                          self._values.data_ptr())

    def __repr__(self):
        return f"COO3_gpu(shape={self._dims}, nnz={self._values.numel()})"


class CSF3_gpu:
    """3-mode tensor with three compressed levels: ``CSF3_gpu(dim_i_indices, dim_j_offsets,
    dim_j_indices, dim_k_offsets, dim_k_indices, values, shape)``; ``dim_j_offsets`` holds
    ``len(dim_i_indices) + 1`` entries and ``dim_k_offsets`` ``len(dim_j_indices) + 1``
    (src/backend/generate_bindings.cpp:119-143)."""

    __slots__ = ("_i", "_jp", "_j", "_kp", "_k", "_values", "_shape", "_dims")

    def __init__(self, dim_i_indices, dim_j_offsets, dim_j_indices, dim_k_offsets, dim_k_indices, values, shape):
        self._i = _dev_array(dim_i_indices, torch.int32, "dim_i_indices")
        self._jp = _dev_array(dim_j_offsets, torch.int32, "dim_j_offsets")
        self._j = _dev_array(dim_j_indices, torch.int32, "dim_j_indices")
        self._kp = _dev_array(dim_k_offsets, torch.int32, "dim_k_offsets")
        self._k = _dev_array(dim_k_indices, torch.int32, "dim_k_indices")
        self._values = _dev_array(values, torch.float32, "values")
        self._shape = _shape_array(shape, 3)
        self._dims = _dims(self._shape)
        if self._jp.numel() != self._i.numel() + 1 or self._kp.numel() != self._j.numel() + 1:
            raise ValueError("offset arrays must hold one entry more than the level above has coordinates")
        if self._k.numel() != self._values.numel():
            raise ValueError("dim_k_indices and values differ in length")

    dim_i_indices = property(lambda self: self._i)
    dim_j_offsets = property(lambda self: self._jp)
    dim_j_indices = property(lambda self: self._j)
    dim_k_offsets = property(lambda self: self._kp)
    dim_k_indices = property(lambda self: self._k)
    values = property(lambda self: self._values)
    shape = property(_host_shape)

    @property
    def device(self):
        return self._values.device

    def _struct(self) -> Csf3Struct:
        dims = (C.c_int32 * 3)(*self._dims)
        return Csf3Struct(dims, self._i.numel(), self._j.numel(), self._k.numel(), self._i.data_ptr(),
                          self._jp.data_ptr(), self._j.data_ptr(), self._kp.data_ptr(), self._k.data_ptr(),
                          self._values.data_ptr())

    def __repr__(self):
        return (f"CSF3_gpu(shape={self._dims}, levels=({self._i.numel()}, "
                f"{self._j.numel()}, {self._k.numel()}))")


def gpu_coo3d_add_f32(a: COO3_gpu, b: COO3_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> COO3_gpu:
    """Z = A + B over sorted unique (i, j, k) coordinates."""
    return _native.coo3d_add(a, b)


def gpu_csf_add_f32(a: CSF3_gpu, b: CSF3_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> CSF3_gpu:
    """Z = A + B for CSF3 operands."""
    return _native.csf_add(a, b)


# ---- the rest of the element-wise family: 2-D COO, DCSR, inner products, masked SpGEMM ----

class COO_gpu:
    """2-D coordinate list sorted by (i, j): ``COO_gpu(dim_i_indices, dim_j_indices, values, shape)``."""

    __slots__ = ("_i", "_j", "_values", "_shape", "_dims")

    def __init__(self, dim_i_indices, dim_j_indices, values, shape):
        self._i = _dev_array(dim_i_indices, torch.int32, "dim_i_indices")
        self._j = _dev_array(dim_j_indices, torch.int32, "dim_j_indices")
        self._values = _dev_array(values, torch.float32, "values")
        self._shape = _shape_array(shape, 2)
        self._dims = _dims(self._shape)
        if not (self._i.numel() == self._j.numel() == self._values.numel()):
            raise ValueError("coordinate arrays and values differ in length")

    dim_i_indices = property(lambda self: self._i)
    dim_j_indices = property(lambda self: self._j)
    values = property(lambda self: self._values)
    shape = property(_host_shape)

    @property
    def device(self):
        return self._values.device

    def __repr__(self):
        return f"COO_gpu(shape={self._dims}, nnz={self._values.numel()})"


class DCSR_gpu:
    """CSR with a compressed row level: ``DCSR_gpu(dim_i_indices, dim_j_offsets, dim_j_indices, values,
    shape)``; ``dim_i_indices`` lists the rows that hold entries, ``dim_j_offsets`` has one entry more."""

    __slots__ = ("_i", "_jp", "_j", "_values", "_shape", "_dims")

    def __init__(self, dim_i_indices, dim_j_offsets, dim_j_indices, values, shape):
        self._i = _dev_array(dim_i_indices, torch.int32, "dim_i_indices")
        self._jp = _dev_array(dim_j_offsets, torch.int32, "dim_j_offsets")
        self._j = _dev_array(dim_j_indices, torch.int32, "dim_j_indices")
        self._values = _dev_array(values, torch.float32, "values")
        self._shape = _shape_array(shape, 2)
        self._dims = _dims(self._shape)
        if self._jp.numel() != self._i.numel() + 1:
            raise ValueError("dim_j_offsets must hold one entry more than dim_i_indices")
        if self._j.numel() != self._values.numel():
            raise ValueError("dim_j_indices and values differ in length")

    dim_i_indices = property(lambda self: self._i)
    dim_j_offsets = property(lambda self: self._jp)
    dim_j_indices = property(lambda self: self._j)
    values = property(lambda self: self._values)
    shape = property(_host_shape)

    @property
    def device(self):
        return self._values.device

    def __repr__(self):
        return f"DCSR_gpu(shape={self._dims}, rows_stored={self._i.numel()}, nnz={self._values.numel()})"


class Scalar_gpu:
    """Result of a full reduction: ``values`` is a one-element float32 CUDA tensor."""

    __slots__ = ("_values",)

    def __init__(self, values):
        self._values = _dev_array(values, torch.float32, "values")

    values = property(lambda self: self._values)

    @property
    def device(self):
        return self._values.device


def gpu_coo_add_f32(a: COO_gpu, b: COO_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> COO_gpu:
    """Z = A + B over sorted unique (i, j) lists."""
    return _native.coo_add(a, b)


def gpu_coo_mul_f32(a: COO_gpu, b: COO_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> COO_gpu:
    """Z = A .* B over sorted unique (i, j) lists."""
    return _native.coo_mul(a, b)


def gpu_coo_csr_add_f32(a: CSR_gpu, b: COO_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> CSR_gpu:
    """Z = A + B with A in CSR and B a coordinate list; the result is CSR."""
    return _native.coo_csr_add(a, b)


def gpu_dcsr_add_f32(a: DCSR_gpu, b: DCSR_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> DCSR_gpu:
    """Z = A + B for DCSR operands."""
    return _native.dcsr_add(a, b)


def gpu_dcsr_mul_f32(a: DCSR_gpu, b: DCSR_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> DCSR_gpu:
    """Z = A .* B for DCSR operands; a row both operands store stays, even with no common column."""
    return _native.dcsr_mul(a, b)


def gpu_dcsr_mul_without_recursive_partitioning_f32(a: DCSR_gpu, b: DCSR_gpu, num_blocks: int = 256,
                                                    threads_per_block: int = 256) -> DCSR_gpu:
    """The reference emits the DCSR product twice to compare two partitioning strategies of its code
    generator (compiler.cpp:128-133); both compute the same tensor, and so does this alias."""
    return gpu_dcsr_mul_f32(a, b, num_blocks, threads_per_block)


def gpu_inner_prod_f32(a: CSF3_gpu, b: CSF3_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> Scalar_gpu:
    """sum_ijk a_ijk * b_ijk for CSF3 operands."""
    return _native.inner_prod(a, b)


def gpu_inner_prod_coo_f32(a: COO3_gpu, b: COO3_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> Scalar_gpu:
    """sum_ijk a_ijk * b_ijk for COO3 operands."""
    return _native.inner_prod_coo(a, b)


def gpu_sssmm_f32(a: CSR_gpu, b: CSR_gpu, c: CSR_gpu, num_blocks: int = 256, threads_per_block: int = 256) -> CSR_gpu:
    """Z_ik = sum_j a_ij * b_jk * c_ik on the positions C stores and a product reaches (masked SpGEMM,
    compiler.cpp:150-153): one fused pass in which the mask drives the accumulation."""
    return _native.sssmm(a, b, c)


_native.bind((CSR_gpu, COO_gpu, DCSR_gpu, COO3_gpu, CSF3_gpu, Scalar_gpu), _capi.check)
