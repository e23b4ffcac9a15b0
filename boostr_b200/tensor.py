"""``QuantTensor``: packed block storage on a CUDA device.

Mirrors ``QuantTensor<R>`` (src/quant/tensor.rs:23-127): raw little-endian blocks as a U8
buffer, the block format, and the LOGICAL element shape.  Blocks run along the last axis.
"""
from __future__ import annotations

import warnings
from typing import Sequence

import numpy as np
import torch

from .format import QuantError, QuantFormat

_hostops = None


class _PythonForms:
    """Stands in for the compiled entry points where they are not built: every call is declined and takes its Python form,
    which enters the same kernels with 10 us more host time."""

    @staticmethod
    def _decline(*args):
        return NotImplemented

    make_ref = quant_matmul = quant_matmul_batch = quant_swiglu = quant_mlp = dequantize = _decline


def hostops():
    """The compiled Python entry points (``csrc/host_ops.cpp``)."""
    global _hostops
    if _hostops is None:
        try:
            from . import _hostops as mod

            if not torch.__version__.startswith(mod.torch_version):
                raise ImportError(f"compiled against torch {mod.torch_version}, running torch {torch.__version__}")
        except ImportError as e:
            warnings.warn(f"the compiled entry points boostr_b200._hostops cannot be used ({e}): calls take their slower Python form. "
                          "Build it with `python -m boostr_b200.build` (needs nvcc and g++; no GPU required)", RuntimeWarning, stacklevel=3)
            mod = _PythonForms
        _hostops = mod
    return _hostops


class QuantTensor:
    def __init__(self, storage: torch.Tensor, fmt: QuantFormat, shape: Sequence[int]):
        own = vars(self)
        own.update(_storage=storage, _format=fmt, _shape=tuple(int(x) for x in shape))
        if storage.is_cuda:  # with the tensor, not in its first call
            own["_ref"] = hostops().make_ref(storage, fmt.format_id, own["_shape"])

    def __getattr__(self, name: str):
        # ``_ref``: what the compiled entry points need of this tensor.  A tensor that is made, read from a file or sharded on the
        # host never asks for them.
        if name != "_ref":
            raise AttributeError(f"{type(self).__name__!r} object has no attribute {name!r}")
        self._ref = ref = hostops().make_ref(self._storage, self._format.format_id, self._shape)
        return ref

    def __setattr__(self, name: str, value) -> None:
        object.__setattr__(self, name, value)
        if name in ("_storage", "_format", "_shape"):
            vars(self).pop("_ref", None)

    def __getstate__(self) -> dict:
        """For copies, pickles and ``torch.save``: ``_ref`` points into this process and to this tensor's storage."""
        return {k: v for k, v in vars(self).items() if k != "_ref"}

    @classmethod
    def from_bytes(cls, data, fmt, shape: Sequence[int], device="cuda") -> "QuantTensor":
        """src/quant/tensor.rs:44-92 — validates the last dimension and the exact byte count."""
        fmt = QuantFormat.parse(fmt)
        shape = tuple(int(x) for x in shape)
        if len(shape) == 0:
            raise QuantError("QuantTensor shape must be non-empty")
        last = shape[-1]
        if last % fmt.block_size:
            raise QuantError(
                f"last dimension {last} is not a multiple of {fmt.name}'s block_size {fmt.block_size}")
        numel = int(np.prod(shape, dtype=np.int64))
        expected = fmt.storage_bytes(numel)
        if isinstance(data, torch.Tensor):
            t = data.reshape(-1)
            if t.dtype != torch.uint8:
                raise QuantError("QuantTensor storage must be uint8")
        else:
            arr = np.frombuffer(data, dtype=np.uint8) if isinstance(data, (bytes, bytearray, memoryview)) else \
                np.ascontiguousarray(data, dtype=np.uint8).reshape(-1)
            t = torch.from_numpy(arr.copy() if not arr.flags.writeable else arr)
        if t.numel() != expected:
            raise QuantError(
                f"expected {expected} bytes for {fmt.name} with {numel} elements, got {t.numel()} bytes")
        t = t.to(device).contiguous()
        if t.data_ptr() % 16:  # torch's allocator hands out 512-byte aligned blocks; views may not be
            t = t.clone()
        return cls(t, fmt, shape)

    # accessors: src/quant/tensor.rs:95-127
    @property
    def format(self) -> QuantFormat:
        return self._format

    @property
    def shape(self) -> tuple:
        return self._shape

    def numel(self) -> int:
        return int(np.prod(self._shape, dtype=np.int64))

    def num_blocks(self) -> int:
        return self.numel() // self._format.block_size

    def storage_bytes(self) -> int:
        return self.num_blocks() * self._format.block_bytes

    @property
    def device(self) -> torch.device:
        return self._storage.device

    @property
    def storage(self) -> torch.Tensor:
        return self._storage
