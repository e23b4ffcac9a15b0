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


def _tensor():
    return QuantTensor.from_bytes(synth.weight_bytes("Q6_K", synth.rng_for(2), 6, 512), "Q6_K", (6, 512), device="cpu")


def _same(a, b):
    return a.format is b.format and a.shape == b.shape and torch.equal(a.storage, b.storage)


@pytest.mark.parametrize("used", [False, True])
def test_copied_and_saved(used):
    """Also a tensor that a compiled call has used, whose handle of native memory stays behind."""
    qt = _tensor()
    if used:
        qt._ref = lambda: None  # like the real handle, nothing that can be copied or saved
    lin = QuantLinear(qt, torch.arange(6.0))
    deep = copy.deepcopy(qt)
    assert _same(deep, qt) and deep.storage.data_ptr() != qt.storage.data_ptr()
    flat = copy.copy(qt)
    assert _same(flat, qt) and flat.storage.data_ptr() == qt.storage.data_ptr()
    for other in (pickle.loads(pickle.dumps(qt)), pickle.loads(pickle.dumps(lin)).weight, copy.deepcopy(lin).weight):
        assert _same(other, qt)
    f = io.BytesIO()
    torch.save({"w": qt}, f)
    f.seek(0)
    assert _same(torch.load(f, weights_only=False)["w"], qt)
    assert all("_ref" not in vars(x) for x in (deep, flat))
