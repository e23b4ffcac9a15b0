"""The K-quant kernel for 9 ... 63 activation rows (csrc/kquant_few.cu) against the CPU oracle: the CPU's bits at every K, also
where a cluster shares a tile (blocks are added in K order)."""
import os

import numpy as np
import pytest

from boostr_b200 import synth
from boostr_b200.format import QuantFormat as F
from boostr_b200.tensor import QuantTensor
from util import describe_mismatch, kq_tile_rows, rel_err, seed_of

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# tiles of 16, 32, 48 activation rows and two of them, one and several blocks, clusters of 2, 4, 8 and whole tiles, weight rows
# around multiples of 128, Q6_K rows of every alignment
SHAPES = [(17, 1, 256), (18, 129, 512), (31, 127, 768), (20, 1000, 4096), (17, 256, 1280), (32, 2500, 2048), (33, 300, 3840), (48, 1300, 4096),
          (49, 128, 512), (63, 4100, 1024), (19, 20000, 512), (32, 19100, 256), (40, 19000, 1536), (37, 700, 14336), (24, 4096, 4352), (63, 900, 8192), (9, 13825, 5120), (16, 14336, 2048),
          (37, 9216, 5120), (33, 5120, 5120), (63, 3072, 4864), (40, 1024, 4608), (17, 400, 2304), (47, 2000, 8448), (48, 130, 512), (18, 128, 768)]


@pytest.mark.parametrize("fmt", ["Q4_K", "Q5_K", "Q6_K"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_products(oracle, fmt, m, n, k):
    from boostr_b200 import ops

    rng = synth.rng_for(101, seed_of(fmt, m, n, k))
    act = synth.activations(rng, m, k)
    act[m // 2] *= 1e-3  # rows of different scale
    act[0, :256] = 0.0   # a block without a maximum
    w = synth.weight_bytes(fmt, rng, n, k)
    guard = 4096
    flat = torch.full((2 * guard + m * n,), 4242.0, device="cuda")
    out = flat[guard:guard + m * n].view(m, n)
    x, qt = torch.from_numpy(act).cuda(), QuantTensor.from_bytes(w, F[fmt], (n, k), device="cuda")
    ops.quant_matmul(x, qt, out=out)
    ops.check_device_status()
    got = out.cpu().numpy()
    assert (flat[:guard] == 4242.0).all() and (flat[guard + m * n:] == 4242.0).all(), "guard regions were written"
    want = oracle.quant_matmul(fmt, act, w, n, threads=os.cpu_count() or 8)
    if m > 16 or kq_tile_rows(fmt, m, n, k) > 0:
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), describe_mismatch(got, want)
    else:  # mma.sync is expected to be faster: its chunks of K are added as sums
        assert rel_err(got, want)[0] <= 2e-6, describe_mismatch(got, want)
    for _ in range(20):
        again = ops.quant_matmul(x, qt)
    assert torch.equal(again.view(torch.int32), out.view(torch.int32))
    ops.check_device_status()


@pytest.mark.parametrize("fmt", ["Q4_K", "Q5_K", "Q6_K"])
@pytest.mark.parametrize("m,n,k", [(17, 64, 28672), (20, 130, 28672), (32, 256, 28672), (33, 100, 28672), (63, 1, 65536), (17, 400, 65536)])
def test_few_weight_rows_of_long_k(oracle, fmt, m, n, k):
    """Too few tiles for the chip: mma.sync shares K out over all of it, and its chunks of K are added as sums."""
    from boostr_b200 import ops

    assert kq_tile_rows(fmt, m, n, k) == -1
    rng = synth.rng_for(103, seed_of(fmt, m, n, k))
    act = synth.activations(rng, m, k)
    w = synth.weight_bytes(fmt, rng, n, k)
    got = ops.quant_matmul(torch.from_numpy(act).cuda(), QuantTensor.from_bytes(w, F[fmt], (n, k), device="cuda")).cpu().numpy()
    ops.check_device_status()
    want = oracle.quant_matmul(fmt, act, w, n, threads=os.cpu_count() or 8)
    assert rel_err(got, want)[0] <= 2e-6, describe_mismatch(got, want)


@pytest.mark.parametrize("fmt", ["Q4_K", "Q5_K", "Q6_K"])
@pytest.mark.parametrize("fill", [0xFF, 0x00, 0xF0, 0x0F, 0x80, 0x7F])
def test_largest_sums(oracle, fmt, fill):
    """Every code, scale and min at an end of its range, activations of one sign and of alternating ones."""
    from boostr_b200 import ops

    m, n, k = 48, 140, 1024
    w = np.full((n * k // 256, F[fmt].block_bytes), fill, np.uint8)
    for at in (208,) if fmt == "Q6_K" else (0, 2):
        w[:, at:at + 2] = np.frombuffer(np.array([1.0], np.float16).tobytes(), np.uint8)
    act = np.ones((m, k), np.float32)
    act[1::3] = -1.0
    act[2::3, ::2] = -1.0
    w = w.reshape(-1)
    for rows in (20, m):
        got = ops.quant_matmul(torch.from_numpy(act[:rows]).cuda(), QuantTensor.from_bytes(w, F[fmt], (n, k), device="cuda")).cpu().numpy()
        want = oracle.quant_matmul(fmt, act[:rows], w, n, threads=4)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), describe_mismatch(got, want)
    ops.check_device_status()


@pytest.mark.parametrize("fmt", ["Q4_K", "Q5_K", "Q6_K"])
@pytest.mark.parametrize("m,n,k", [(18, 65, 512), (24, 9500, 1280), (33, 500, 4096), (20, 1000, 5120), (12, 5632, 2048), (37, 4500, 5120), (63, 2000, 4608), (19, 100, 2304)])
def test_swiglu(fmt, m, n, k):
    """silu(gate) * up of the two products, to the rounding of one f32 expression."""
    from boostr_b200 import ops

    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed_of(fmt, m, n, k))
    g, u = synth.device_weight(fmt, n, k, gen), synth.device_weight(fmt, n, k, gen)
    x = torch.randn(m, k, device="cuda", generator=gen)
    a, b = ops.quant_matmul(x, g).double(), ops.quant_matmul(x, u).double()
    got = ops.quant_swiglu(x, g, u)
    ops.check_device_status()
    want = a / (1 + torch.exp(-a)) * b
    # the same products; expf within 2 ulp, three more roundings (4 * 2^-23)
    assert ((got.double() - want).abs() <= 5e-7 * want.abs() + 1e-36 * b.abs()).all()


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("m", [17, 24, 32, 33, 48, 63])
def test_batch_shares_one_image(m, reverse):
    """All K-quant weights of a batch of 17 ... 63 rows read one image of the activations, whatever their order, and give the bits of
    separate calls."""
    from boostr_b200 import ops

    gen = torch.Generator(device="cuda")
    gen.manual_seed(m)
    k = 1536
    specs = [("Q4_K", 1500), ("Q6_K", 300), ("Q2_K", 300), ("Q5_K", 2100), ("Q3_K", 200), ("Q4_K", 129), ("Q6_K", 2049)]
    ws = [synth.device_weight(fmt, n, k, gen) for fmt, n in (reversed(specs) if reverse else specs)]
    x = torch.randn(m, k, device="cuda", generator=gen)
    want = [ops.quant_matmul(x, w) for w in ws]
    before = ops.launch_count()
    got = ops.quant_matmul_batch(x, ws)
    assert ops.launch_count() - before == 1 + len(ws)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    ops.check_device_status()


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("m", [9, 13, 16])
def test_batch_that_changes_the_kernel(m, reverse):
    """At 9 ... 16 rows the weights of a batch go to this kernel and to mma.sync in turn: each finds its own image in the scratch."""
    from boostr_b200 import ops

    gen = torch.Generator(device="cuda")
    gen.manual_seed(m)
    k = 2048
    specs = [("Q5_K", 14336), ("Q5_K", 1024), ("Q6_K", 14336), ("Q4_K", 1024), ("Q2_K", 300), ("Q5_K", 14336), ("Q6_K", 512), ("Q4_K", 200)]
    ws = [synth.device_weight(fmt, n, k, gen) for fmt, n in (reversed(specs) if reverse else specs)]
    tiles = [kq_tile_rows(w.format.name, m, *w.shape) for w in ws if w.format is not F.Q2_K]
    assert max(tiles) > 0 and min(tiles) < 0
    x = torch.randn(m, k, device="cuda", generator=gen)
    want = [ops.quant_matmul(x, w) for w in ws]
    for a, b in zip(ops.quant_matmul_batch(x, ws), want):
        assert torch.equal(a, b)
    ops.check_device_status()


@pytest.mark.parametrize("fmt", ["Q4_K", "Q5_K", "Q6_K"])
@pytest.mark.parametrize("m,n,k", [(24, 700, 2048), (37, 1300, 5120), (63, 19000, 256), (17, 1000, 768)])
def test_16_bit_activations_and_results(oracle, fmt, m, n, k):
    from boostr_b200 import ops

    assert kq_tile_rows(fmt, m, n, k) > 0
    rng = synth.rng_for(102, seed_of(fmt, m, n, k))
    x = torch.from_numpy(synth.activations(rng, m, k)).cuda().to(torch.bfloat16)
    w = synth.weight_bytes(fmt, rng, n, k)
    qt = QuantTensor.from_bytes(w, F[fmt], (n, k), device="cuda")
    got = ops.quant_matmul(x, qt, out_dtype=torch.float32)
    want = oracle.quant_matmul(fmt, x.float().cpu().numpy(), w, n, threads=os.cpu_count() or 8)
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32)), describe_mismatch(got.cpu().numpy(), want)
    for dt in (torch.bfloat16, torch.float16):  # one rounding of the f32 results
        assert torch.equal(ops.quant_matmul(x, qt, out_dtype=dt), got.to(dt))
    ops.check_device_status()


def test_more_weight_rows_than_2_to_the_22():
    """The last rows of a weight of more than 2^22 rows have the bits that they have in a weight of their own."""
    from boostr_b200 import ops

    m, n, k, tail = 17, (1 << 22) + 200, 256, 300
    gen = torch.Generator(device="cuda")
    gen.manual_seed(22)
    w = synth.device_weight("Q4_K", n, k, gen)
    x = torch.randn(m, k, device="cuda", generator=gen)
    block = F.Q4_K.block_bytes
    part = QuantTensor(w.storage[(n - tail) * block:n * block].clone(), w.format, (tail, k))
    assert torch.equal(ops.quant_matmul(x, w)[:, n - tail:], ops.quant_matmul(x, part))
    ops.check_device_status()
