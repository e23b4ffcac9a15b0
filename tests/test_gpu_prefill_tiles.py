"""The tensor-core path at the lines of its tile rule (64, 128, 192 or 256 activation rows a tile): either side of each row
count, partial tiles, whole and K-split tiles, against the same bf16 operands in f32 (the bound of the existing cases)."""
import numpy as np
import pytest

from boostr_b200 import synth
from test_gpu_parity import _bf16_reference, _prepared_act, _qt
from util import describe_mismatch, rel_err, seed_of

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("fmt", ["Q4_K", "Q6_K", "Q8_0"])
@pytest.mark.parametrize("m,n,k", [(255, 300, 1024), (256, 300, 2048), (257, 20000, 256), (300, 9000, 1024), (384, 8193, 512), (385, 9000, 512),
                                   (384, 1024, 2048), (900, 130, 4096), (1023, 1024, 512), (1024, 1024, 512),
                                   (256, 4096, 4096), (256, 4000, 4352), (512, 1000, 6144), (300, 700, 6400), (700, 200, 8448)])
def test_tile_rule(oracle, fmt, m, n, k):
    from boostr_b200 import ops

    rng = synth.rng_for(95, seed_of(fmt, m, n, k))
    act = synth.activations(rng, m, k)
    qt = _qt(fmt, synth.weight_bytes(fmt, rng, n, k), n, k)
    guard = 4096
    flat = torch.full((2 * guard + m * n,), 777.0, device="cuda")
    got = ops.quant_matmul(torch.from_numpy(act).cuda(), qt, out=flat[guard:guard + m * n].view(m, n)).cpu().numpy()
    ops.check_device_status()
    assert torch.all(flat[:guard] == 777.0) and torch.all(flat[guard + m * n:] == 777.0)
    ref = _bf16_reference(ops, _prepared_act(oracle, fmt, act), qt)
    assert np.isfinite(got).all() and rel_err(got, ref)[0] <= 2e-5, describe_mismatch(got, ref)
