"""``QuantTensor`` on the host: it can be made, read from a file, copied, saved and sent without the compiled entry points."""
import copy
import io
import os
import pickle
import subprocess
import sys

import pytest
import torch

from boostr_b200 import synth
from boostr_b200.linear import QuantLinear
from boostr_b200.tensor import QuantTensor

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_host_use_needs_no_compiled_entry_points(tmp_path):
    """A tree in which ``_hostops`` cannot be imported: tensors are made and a file is read all the same."""
    code = """
import sys
sys.modules["boostr_b200._hostops"] = None
from boostr_b200 import gguf, synth, tensor
qt = tensor.QuantTensor.from_bytes(synth.weight_bytes("Q4_K", synth.rng_for(1), 8, 512), "Q4_K", (8, 512), device="cpu")
assert qt.shape == (8, 512) and qt.storage_bytes() == qt.storage.numel()
assert not hasattr(qt, "no_such_attribute")
import warnings, torch
from boostr_b200 import ops
from boostr_b200.format import QuantError
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    for call in (lambda: ops.quant_matmul(torch.zeros(1, 512), qt), lambda: ops.dequantize(qt), lambda: ops.quant_swiglu(torch.zeros(1, 256), qt, qt)):
        try:
            call()
        except QuantError:
            pass  # "must live on a CUDA device", "dimension mismatch": the operators' own words
        else:
            raise SystemExit("a host tensor was taken")
assert len(seen) == 1 and "slower Python form" in str(seen[0].message)
"""
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, check=True)
