"""Q2_K / Q3_K products at the edges of their kernels' tiles, bit for bit against the CPU oracle (integer sums, blocks added
in K order): row counts around the multiples of 8 and 16 of the mma.sync kernel and of 16 ... 128 of the tensor-core
kernel, partial row tiles, one block and odd block counts (rows of every alignment), more tiles than SMs, long K."""
import os

import numpy as np
import pytest

from boostr_b200 import synth
from boostr_b200.format import QuantFormat as F
from boostr_b200.tensor import QuantTensor
from util import describe_mismatch, seed_of

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("fmt", ["Q2_K", "Q3_K"])
@pytest.mark.parametrize("m,n,k", [
    (1, 17, 256), (7, 2400, 1280), (8, 16, 3840), (3, 500, 14336), (1, 9000, 4352),
    (9, 129, 1280), (16, 128, 256), (17, 100, 768), (32, 4736, 512), (24, 31, 14336),
    (33, 128, 256), (64, 1, 1280), (100, 1000, 768), (128, 257, 512), (129, 130, 1280), (300, 4097, 256), (512, 1024, 2304), (70, 200, 14336)])
def test_bit_identical(oracle, fmt, m, n, k):
    from boostr_b200 import ops

    rng = synth.rng_for(93, seed_of(fmt, m, n, k))
    act = synth.activations(rng, m, k)
    act[m // 2] *= 1e-3  # rows of different scale
    act[0, :256] = 0.0   # a block without a maximum
    w = synth.weight_bytes(fmt, rng, n, k)
    guard = 4096
    flat = torch.full((2 * guard + m * n,), 4242.0, device="cuda")
    out = flat[guard:guard + m * n].view(m, n)
    qt = QuantTensor.from_bytes(w, F[fmt], (n, k), device="cuda")
    x = torch.from_numpy(act).cuda()
    ops.quant_matmul(x, qt, out=out)
    ops.check_device_status()
    got = out.cpu().numpy()
    assert (flat[:guard] == 4242.0).all() and (flat[guard + m * n:] == 4242.0).all(), "guard regions were written"
    want = oracle.quant_matmul(fmt, act, w, n, threads=os.cpu_count() or 8)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), describe_mismatch(got, want)
    # both formats of a batch read one activation image; 16-bit results are one rounding of the f32 ones
    pair = ops.quant_matmul_batch(x, [qt, qt], out_dtype=torch.bfloat16)
    for y in pair:
        assert torch.equal(y, out.to(torch.bfloat16))


@pytest.mark.parametrize("fmt", ["Q4_K", "Q5_K"])
@pytest.mark.parametrize("m,n,k", [(17, 9000, 1280), (33, 2050, 512), (37, 4097, 1280), (48, 2100, 768), (49, 20000, 256), (63, 30000, 512)])
def test_two_byte_products_bit_identical(oracle, fmt, m, n, k):
    from boostr_b200 import ops

    rng = synth.rng_for(94, seed_of(fmt, m, n, k))
    act = synth.activations(rng, m, k)
    act[m // 2] *= 1e-3
    act[0, :256] = 0.0
    w = synth.weight_bytes(fmt, rng, n, k)
    guard = 4096
    flat = torch.full((2 * guard + m * n,), 4242.0, device="cuda")
    out = flat[guard:guard + m * n].view(m, n)
    ops.quant_matmul(torch.from_numpy(act).cuda(), QuantTensor.from_bytes(w, F[fmt], (n, k), device="cuda"), out=out)
    ops.check_device_status()
    got = out.cpu().numpy()
    assert (flat[:guard] == 4242.0).all() and (flat[guard + m * n:] == 4242.0).all(), "guard regions were written"
    want = oracle.quant_matmul(fmt, act, w, n, threads=os.cpu_count() or 8)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), describe_mismatch(got, want)


def test_extreme_codes(oracle):
    """Every scale, code and activation at its largest: the integer sums reach their bounds."""
    from boostr_b200 import ops

    m, n, k = 64, 128, 512
    act = np.ones((m, k), np.float32)
    act[1::2] = -1.0
    for fmt, fill in (("Q2_K", 0xFF), ("Q3_K", 0x00), ("Q3_K", 0xFF)):
        blk = F[fmt].block_bytes
        w = np.full((n * k // 256, blk), fill, np.uint8)
        w[:, -4:] = np.frombuffer(np.array([1.0, 1.0], np.float16).tobytes(), np.uint8) if fmt == "Q2_K" else w[:, -4:]
        if fmt == "Q3_K":
            w[:, -2:] = np.frombuffer(np.array([1.0], np.float16).tobytes(), np.uint8)
        w = w.reshape(-1)
        for rows in (4, m):
            got = ops.quant_matmul(torch.from_numpy(act[:rows]).cuda(), QuantTensor.from_bytes(w, F[fmt], (n, k), device="cuda")).cpu().numpy()
            want = oracle.quant_matmul(fmt, act[:rows], w, n, threads=4)
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), describe_mismatch(got, want)
