"""The compiled Python entry points (``csrc/host_ops.cpp``): what they take, what they leave to the Python form, and the scratch
that they share between calls."""
import pytest

from boostr_b200 import synth
from boostr_b200.format import QuantFormat as F
from boostr_b200.tensor import QuantTensor, hostops

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ops():
    from boostr_b200 import ops as o

    assert hostops().__name__ == "boostr_b200._hostops", "the compiled entry points are not built"
    return o


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def test_lists_that_change_during_the_call(ops):
    """The entry points read an attribute of every weight, which may run Python code that shrinks the lists of the call."""
    gen = _gen(1)
    outs = []

    class Shrinking(QuantTensor):
        @property
        def _ref(self):
            del outs[1:], weights[1:]
            return hostops().make_ref(self.storage, self.format.format_id, self.shape)

    base = [synth.device_weight("Q4_K", 64, 256, gen) for _ in range(3)]
    weights = [Shrinking(w.storage, w.format, w.shape) for w in base]
    x = torch.randn(2, 256, device="cuda", generator=gen)
    outs.extend(torch.empty(2, 64, device="cuda") for _ in range(3))
    kept = list(outs)
    got = ops.quant_matmul_batch(x, weights, outs=outs)
    assert len(got) == 3 and all(a is b for a, b in zip(got, kept))
    for y, w in zip(got, base):
        assert torch.equal(y, ops.quant_matmul(x, w))


def test_unknown_format_is_an_error(ops):
    class Fmt:  # Q4_1, which the library does not read
        format_id, block_size, block_bytes, name = 1, 32, 20, "Q4_1"

    qt = QuantTensor(torch.zeros(20 * 8, dtype=torch.uint8, device="cuda"), Fmt(), (8, 32))
    with pytest.raises(RuntimeError, match="unsupported format id 1"):
        ops.dequantize(qt)
    with pytest.raises(RuntimeError, match="unsupported format id 1"):
        ops.quant_matmul(torch.zeros(1, 32, device="cuda"), qt)


def test_replaced_storage_is_read(ops):
    """A tensor whose storage is exchanged after a call: the next call reads the new one."""
    gen = _gen(2)
    a, b = (synth.device_weight("Q4_K", 64, 512, gen) for _ in range(2))
    x = torch.randn(3, 512, device="cuda", generator=gen)
    want = ops.quant_matmul(x, b), ops.dequantize(b)
    ops.quant_matmul(x, a), ops.dequantize(a)
    a._storage = b.storage.clone()
    assert torch.equal(ops.quant_matmul(x, a), want[0]) and torch.equal(ops.dequantize(a), want[1])


def test_outputs_given_in_part(ops):
    """None among the outputs of a batch: that one is allocated, and returned."""
    gen = _gen(5)
    w = synth.device_weight("Q4_K", 64, 512, gen)
    x = torch.randn(3, 512, device="cuda", generator=gen)
    y = torch.empty(3, 64, device="cuda")
    got = ops.quant_matmul_batch(x, [w, w], outs=[None, y])
    assert got[1] is y and torch.equal(got[0], y) and torch.equal(y, ops.quant_matmul(x, w))
