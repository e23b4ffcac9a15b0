"""A weight written by the kernel before a product in the stream: the product reads what that kernel wrote.

The writer is itself one of the library's kernels, which let the next launch begin early: a long product of a few rows whose
result is the first bytes of the packed weight.  Prompt products (64 rows and more), Q2_K and Q3_K products order all their
reads behind it."""
import pytest

from boostr_b200 import synth
from boostr_b200.format import QuantFormat as F
from boostr_b200.tensor import QuantTensor

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _writer(ops, gen):
    """8 x 128 f32 results from a reduction of 262144: a few CTAs for some hundred microseconds."""
    wx = torch.randn(8, 262144, device="cuda", generator=gen)
    ww = synth.device_weight("Q3_K", 128, 262144, gen)
    return lambda dst: ops.quant_matmul(wx, ww, out=dst)


@pytest.mark.parametrize("fmt,m,n,k,act", [
    ("Q4_K", 64, 128, 256, "f32"), ("Q4_K", 300, 500, 2048, "bf16"), ("Q5_K", 64, 128, 512, "f32"), ("Q6_K", 64, 130, 256, "f32"),
    ("Q6_K", 64, 128, 2048, "f32"), ("Q8_0", 64, 128, 256, "f32"), ("Q8_0", 64, 128, 256, "bf16"), ("Q4_0", 100, 200, 512, "bf16"),
    ("Q5_0", 64, 64, 64, "bf16"), ("Q2_K", 1, 64, 256, "f32"), ("Q3_K", 12, 100, 512, "f32"), ("Q2_K", 512, 4096, 1024, "f32"),
    ("Q3_K", 512, 4096, 2048, "bf16")])
def test_product_reads_what_the_kernel_before_it_wrote(fmt, m, n, k, act):
    from boostr_b200 import ops

    gen = torch.Generator(device="cuda")
    gen.manual_seed(11)
    write = _writer(ops, gen)
    qt = synth.device_weight(fmt, n, k, gen)
    head = qt.storage[:4096] if qt.storage.numel() >= 4096 else None
    if head is None:  # a packed weight shorter than the writer's result: its own bytes are the front of a longer buffer
        buf = torch.zeros(4096, dtype=torch.uint8, device="cuda")
        qt = QuantTensor(buf[:qt.storage.numel()], F[fmt], (n, k))
        head = buf
    dst = head.view(torch.float32).view(8, 128)
    x = torch.randn(m, k, device="cuda", generator=gen).to(torch.float32 if act == "f32" else torch.bfloat16)
    got, want, stale = (torch.empty(m, n, device="cuda") for _ in range(3))
    for _ in range(2):  # the first pass also loads the kernels
        head.zero_()
        ops.quant_matmul(x, qt, out=stale)
        torch.cuda.synchronize()
        write(dst)
        ops.quant_matmul(x, qt, out=got)
        torch.cuda.synchronize()
        ops.quant_matmul(x, qt, out=want)
        torch.cuda.synchronize()
    ops.check_device_status()
    assert not torch.equal(want.view(torch.int32), stale.view(torch.int32)), "the written bytes do not matter"
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("first", ["Q5_K", "Q3_K"])
@pytest.mark.parametrize("fmt,n", [("Q2_K", 300), ("Q3_K", 9000)])
def test_later_product_of_a_batch_reads_what_the_kernel_before_the_batch_wrote(first, fmt, n):
    """The first product of the batch (of few tiles, so that the second finds room beside it) may start ahead of the writer's end."""
    from boostr_b200 import ops

    gen = torch.Generator(device="cuda")
    gen.manual_seed(12)
    write = _writer(ops, gen)
    m, k = 20, 512
    head, qt = synth.device_weight(first, 4100, k, gen), synth.device_weight(fmt, n, k, gen)
    dst = qt.storage[:4096].view(torch.float32).view(8, 128)
    x = torch.randn(m, k, device="cuda", generator=gen)
    outs = [torch.empty(m, w.shape[0], device="cuda") for w in (head, qt)]
    for _ in range(2):
        qt.storage[:4096].zero_()
        torch.cuda.synchronize()
        write(dst)
        ops.quant_matmul_batch(x, [head, qt], outs=outs)
        torch.cuda.synchronize()
        want = ops.quant_matmul(x, qt)
    ops.check_device_status()
    assert torch.equal(outs[1].view(torch.int32), want.view(torch.int32))
