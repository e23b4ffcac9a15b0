"""Shared helpers for the parity tests."""
import numpy as np


def rel_err(got: np.ndarray, ref: np.ndarray):
    """(max|got-ref| / max|ref|, rms(got-ref) / rms(ref)) — the error measure used for every
    matmul tolerance in this suite.  Element-wise relative error is meaningless here because
    outputs cross zero."""
    got = np.asarray(got, dtype=np.float64)
    ref = np.asarray(ref, dtype=np.float64)
    den = max(np.abs(ref).max(), 1e-30)
    rms = max(np.sqrt((ref ** 2).mean()), 1e-30)
    d = got - ref
    return float(np.abs(d).max() / den), float(np.sqrt((d ** 2).mean()) / rms)


def describe_mismatch(got: np.ndarray, ref: np.ndarray, limit: int = 8) -> str:
    got = np.asarray(got)
    ref = np.asarray(ref)
    bad = np.argwhere(~np.isclose(got, ref, rtol=1e-4, atol=1e-6 * max(np.abs(ref).max(), 1e-30)))
    lines = [f"{len(bad)} of {got.size} elements differ; first {min(limit, len(bad))}:"]
    for idx in bad[:limit]:
        t = tuple(int(i) for i in idx)
        lines.append(f"  {t}: got {got[t]!r} want {ref[t]!r}")
    return "\n".join(lines)


def seed_of(*parts) -> int:
    """Deterministic small integer from test parameters (Python's str hash is salted per process)."""
    import zlib

    return zlib.crc32(repr(parts).encode()) % 1000


def kq_tile_rows(fmt, m, n, k):
    """Activation rows of the tensor-core tile that the library's own rule gives a K-quant product (0: kernel for few rows, -1: another
    path)."""
    import ctypes

    import torch

    from boostr_b200 import _cabi
    from boostr_b200.format import QuantFormat

    f = _cabi.lib().b200q_kq_tile_rows
    f.restype, f.argtypes = ctypes.c_int, [ctypes.c_int, ctypes.c_size_t, ctypes.c_size_t, ctypes.c_size_t, ctypes.c_int]
    return f(QuantFormat[fmt].format_id, m, k, n, torch.cuda.get_device_properties(0).multi_processor_count)
