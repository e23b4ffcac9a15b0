"""The integer tensor-core products of the K-quants, bit for bit against the CPU oracle (integer sums, blocks added in K order): Q2_K and
Q3_K (csrc/kquant_i8.cu), Q4_K and Q5_K with 17 ... 63 rows (csrc/kquant_few.cu).
``test_bit_identical``: Q2_K / Q3_K around the multiples of 8 and 16 rows of the mma.sync kernel (which takes all of its shapes but
the two of 300 and 512 rows), partial row tiles, one block and odd block counts (rows of every alignment), long K.
``test_weight_tiles_by_tma``: the tensor-core kernel on tiles of 16 ... 128 rows, held to the rule that picks them."""
import os

import numpy as np
import pytest

from boostr_b200 import synth
from boostr_b200.format import QuantFormat as F
from boostr_b200.tensor import QuantTensor
from util import describe_mismatch, kq_tile_rows, seed_of

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


@pytest.mark.parametrize("fmt,m,n,k,tile", [
    ("Q2_K", 48, 18900, 1024, 48), ("Q2_K", 112, 18900, 1024, 112), ("Q2_K", 128, 18900, 2048, 128), ("Q2_K", 129, 18900, 1024, 80),
    ("Q2_K", 300, 5001, 4096, 112), ("Q2_K", 512, 4096, 2048, 128),
    ("Q3_K", 24, 18900, 2048, 32), ("Q3_K", 112, 18900, 2048, 112), ("Q3_K", 128, 18900, 2048, 128), ("Q3_K", 300, 4001, 2048, 80),
    ("Q3_K", 512, 4096, 4096, 128), ("Q4_K", 33, 18900, 2048, 48), ("Q4_K", 48, 14336, 2048, 48), ("Q4_K", 63, 20000, 1024, 32),
    ("Q4_K", 40, 18900, 256, 48), ("Q5_K", 17, 2050, 256, 16), ("Q5_K", 20, 18900, 2048, 32), ("Q5_K", 37, 13825, 5120, 48), ("Q5_K", 48, 18900, 256, 48)])
def test_weight_tiles_by_tma(oracle, fmt, m, n, k, tile):
    """Rows that are a multiple of 16 bytes, as in every real matrix: the packed blocks come by TMA.  Whole and partial tiles,
    every CTA with one unit or several, one block of K up to twenty; the ring of packed blocks must end with the work (a
    bounded wait that ran out would show in the status word), also over many launches of the shortest work."""
    from boostr_b200 import ops

    assert kq_tile_rows(fmt, m, n, k) == tile and k // 256 * F[fmt].block_bytes % 16 == 0
    rng = synth.rng_for(96, seed_of(fmt, m, n, k))
    act = synth.activations(rng, m, k)
    w = synth.weight_bytes(fmt, rng, n, k)
    x, qt = torch.from_numpy(act).cuda(), QuantTensor.from_bytes(w, F[fmt], (n, k), device="cuda")
    out = ops.quant_matmul(x, qt)
    again = torch.empty_like(out)
    for _ in range(200 if k == 256 else 3):
        ops.quant_matmul(x, qt, out=again)
    ops.check_device_status()
    assert torch.equal(out.view(torch.int32), again.view(torch.int32))
    got = out.cpu().numpy()
    want = oracle.quant_matmul(fmt, act, w, n, threads=os.cpu_count() or 8)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), describe_mismatch(got, want)


@pytest.mark.parametrize("fmt", ["Q4_K", "Q5_K"])
@pytest.mark.parametrize("m,n,k", [(17, 9000, 1280), (33, 2050, 512), (37, 4097, 1280), (48, 2100, 768), (49, 20000, 256), (63, 30000, 512)])
def test_q4_k_and_q5_k_bit_identical(oracle, fmt, m, n, k):
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


def test_batch_shares_one_image():
    """The Q2_K, Q3_K and Q5_K weights of a batch read one image of the activations."""
    from boostr_b200 import ops

    gen = torch.Generator(device="cuda")
    gen.manual_seed(7)
    m, k = 37, 1280
    ws = [synth.device_weight(fmt, n, k, gen) for fmt, n in (("Q5_K", 4097), ("Q3_K", 300), ("Q2_K", 300), ("Q5_K", 4100))]
    assert all(kq_tile_rows(w.format.name, m, *w.shape) >= 0 for w in ws)
    x = torch.randn(m, k, device="cuda", generator=gen)
    want = [ops.quant_matmul(x, w) for w in ws]
    before = ops.launch_count()
    got = ops.quant_matmul_batch(x, ws)
    assert ops.launch_count() - before == 1 + len(ws)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


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


@pytest.mark.parametrize("fmt,m,n,k", [("Q2_K", 512, 4096, 1024), ("Q3_K", 512, 4096, 2048), ("Q4_K", 48, 14336, 1024), ("Q5_K", 48, 14336, 1024),
                                       ("Q5_K", 20, 4100, 512)])
@pytest.mark.parametrize("fill", [0xFF, 0x00, 0xF0, 0x0F])
def test_extreme_codes_in_tiles(oracle, fmt, m, n, k, fill):
    """The same in the tensor-core kernel: every code, scale and min at an end of its range, activations of one sign and of
    alternating ones, so that the sums reach their bounds."""
    from boostr_b200 import ops

    assert kq_tile_rows(fmt, m, n, k) > 0
    w = np.full((n * k // 256, F[fmt].block_bytes), fill, np.uint8)
    one = np.frombuffer(np.array([1.0], np.float16).tobytes(), np.uint8)
    for at in {"Q2_K": (80, 82), "Q3_K": (108,), "Q4_K": (0, 2), "Q5_K": (0, 2)}[fmt]:
        w[:, at:at + 2] = one
    act = np.ones((m, k), np.float32)
    act[1::3] = -1.0
    act[2::3, ::2] = -1.0
    got = ops.quant_matmul(torch.from_numpy(act).cuda(), QuantTensor.from_bytes(w.reshape(-1), F[fmt], (n, k), device="cuda")).cpu().numpy()
    ops.check_device_status()
    want = oracle.quant_matmul(fmt, act, w.reshape(-1), n, threads=os.cpu_count() or 8)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), describe_mismatch(got, want)


@pytest.mark.parametrize("fmt,m,n,k", [("Q2_K", 5, 131, 512), ("Q3_K", 300, 4001, 256), ("Q4_K", 37, 8193, 512), ("Q5_K", 21, 4099, 512), ("Q4_K", 65, 131, 256)])
def test_swiglu_and_its_output(fmt, m, n, k):
    """SwiGLU is silu(gate) * up of the two products; the last kernel takes outputs of any 4-byte alignment, an element count
    that is no multiple of four, and 16-bit results that are one rounding of the f32 ones."""
    from boostr_b200 import ops

    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed_of(fmt, m, n, k))
    g, u = synth.device_weight(fmt, n, k, gen), synth.device_weight(fmt, n, k, gen)
    x = torch.randn(m, k, device="cuda", generator=gen)
    a, b = ops.quant_matmul(x, g).double(), ops.quant_matmul(x, u).double()
    want = a / (1 + torch.exp(-a)) * b
    out = ops.quant_swiglu(x, g, u)
    # expf is within 2 ulp, the sum, the quotient and the product within half a one each: below 4 * 2^-23; past -88 expf overflows
    # and the result is 0 in place of less than 1e-36 |b|
    assert ((out.double() - want).abs() <= 5e-7 * want.abs() + 1e-36 * b.abs()).all()
    for shift in (1, 2, 3):
        buf = torch.full((m * n + 8,), 77.0, device="cuda")
        y = ops.quant_swiglu(x, g, u, out=buf[shift:shift + m * n].view(m, n))
        assert torch.equal(y, out) and (buf[:shift] == 77.0).all() and (buf[shift + m * n:] == 77.0).all()
    for dt in (torch.bfloat16, torch.float16):
        assert torch.equal(ops.quant_swiglu(x, g, u, out_dtype=dt), out.to(dt))
    d = synth.device_weight("Q6_K", 64, 8192, gen)
    if n >= 8192:  # the feed-forward block on these kernels: SwiGLU, then the down product
        g8, u8 = (QuantTensor(t.storage[:F[fmt].storage_bytes(8192 * k)], t.format, (8192, k)) for t in (g, u))
        assert torch.equal(ops.quant_mlp(x, g8, u8, d), ops.quant_matmul(ops.quant_swiglu(x, g8, u8), d))
    ops.check_device_status()
