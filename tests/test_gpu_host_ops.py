"""The compiled Python entry points (``csrc/host_ops.cpp``): what they take, what they leave to the Python form, and the scratch
that they share between calls."""
import threading

import pytest

from boostr_b200 import synth, tensor
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


def _calls(ops):
    """name -> call; the compiled form serves some, leaves some to the Python form and lets some fail."""
    gen = _gen(3)
    w, w2, w6 = (synth.device_weight(f, n, 512, gen) for f, n in (("Q4_K", 96, ), ("Q4_K", 96), ("Q6_K", 40)))
    w8, down = synth.device_weight("Q8_0", 33, 512, gen), synth.device_weight("Q6_K", 50, 256, gen)
    gate, up = synth.device_weight("Q4_K", 256, 512, gen), synth.device_weight("Q4_K", 256, 512, gen)
    vec = synth.device_weight("Q4_K", 1, 1024, gen)
    flat = QuantTensor(vec.storage, vec.format, (1024,))
    on_host = QuantTensor(w.storage.cpu(), w.format, w.shape)
    x = {m: torch.randn(m, 512, device="cuda", generator=gen) for m in (1, 7, 20, 70)}
    y = x[7]
    odd = torch.cat([y.view(-1)[:1], y.view(-1)])[1:].view(7, 512)
    norm = torch.rand(512, device="cuda", generator=gen)
    f32 = dict(dtype=torch.float32, device="cuda")
    c = {}
    for m, a in x.items():
        c[f"matmul {m}"] = lambda a=a: ops.quant_matmul(a, w)
        c[f"matmul {m} bf16"] = lambda a=a: ops.quant_matmul(a.bfloat16(), w8, out_dtype=torch.float16)
        c[f"batch {m}"] = lambda a=a: ops.quant_matmul_batch(a, (w, w6, w8), out_dtype=torch.bfloat16)
        c[f"norm {m}"] = lambda a=a: ops.rmsnorm_quant_matmul_batch(a, norm, 1, [w, w6])
        c[f"swiglu {m}"] = lambda a=a: ops.quant_swiglu(a, w, w2)
        c[f"mlp {m}"] = lambda a=a: ops.quant_mlp(a, gate, up, down)
    c.update({
        "1-D": lambda: ops.quant_matmul(y[0], w), "4-D": lambda: ops.quant_matmul(y.view(1, 7, 1, 512), w), "no rows": lambda: ops.quant_matmul(y[:0], w),
        "no dimension": lambda: ops.quant_matmul(torch.zeros((), device="cuda"), w), "strided": lambda: ops.quant_matmul(x[20][::2], w),
        "transposed": lambda: ops.quant_matmul(y.t().contiguous().t(), w), "misaligned": lambda: ops.quant_mlp(odd, gate, up, down),
        "parameter": lambda: ops.quant_matmul(torch.nn.Parameter(y), w).detach(), "half": lambda: ops.quant_matmul(y.half(), w),
        "bf16 not allowed": lambda: ops.quant_matmul(y.bfloat16(), w, allow_bf16_activation=False), "K": lambda: ops.quant_matmul(y[:, :256].contiguous(), w),
        "host activation": lambda: ops.quant_matmul(y.cpu(), w), "host weight": lambda: ops.quant_matmul(y, on_host), "1-D weight": lambda: ops.quant_matmul(y, flat),
        "f64 result": lambda: ops.quant_matmul(y, w, out_dtype=torch.float64), "integer result": lambda: ops.quant_matmul(y, w, out_dtype=torch.int32),
        "out": lambda: ops.quant_matmul(y, w, out=torch.zeros(7, 96, **f32)), "out shape": lambda: ops.quant_matmul(y, w, out=torch.zeros(7, 95, **f32)),
        "out rows": lambda: ops.quant_matmul(y, w, out=torch.zeros(8, 96, **f32)), "out rank": lambda: ops.quant_matmul(y, w, out=torch.zeros(1, 7, 96, **f32)),
        "out type": lambda: ops.quant_matmul(y, w, out=torch.zeros(7, 96, device="cuda").half()), "out strided": lambda: ops.quant_matmul(y, w, out=torch.zeros(96, 7, **f32).t()),
        "out on host": lambda: ops.quant_swiglu(y, w, w2, out=torch.zeros(7, 96)), "out odd address": lambda: ops.quant_matmul(y, w, out=torch.zeros(7 * 96 + 1, **f32)[1:].view(7, 96)),
        "no weights": lambda: ops.quant_matmul_batch(y, []), "many weights": lambda: ops.quant_matmul_batch(y, [w8] * 17),
        "outs": lambda: ops.quant_matmul_batch(y, [w, w6], outs=(torch.zeros(7, 96, **f32), torch.zeros(7, 40, **f32))),
        "outs long": lambda: ops.quant_matmul_batch(y, [w6], outs=[torch.zeros(7, 40, **f32), None]),
        "outs short": lambda: ops.quant_matmul_batch(y, [w6, w6], outs=[torch.zeros(7, 40, **f32)]),
        "outs partly": lambda: ops.quant_matmul_batch(y, [w6, w6], outs=[None, torch.zeros(7, 40, **f32)]),
        "batch K": lambda: ops.quant_matmul_batch(y, [w, down]), "norm length": lambda: ops.rmsnorm_quant_matmul_batch(y, norm[:256], 1e-5, [w]),
        "norm type": lambda: ops.rmsnorm_quant_matmul_batch(y, norm.bfloat16(), 1e-5, [w]), "norm address": lambda: ops.rmsnorm_quant_matmul_batch(y, torch.cat([norm, norm])[1:513], 1e-5, [w]),
        "norm on host": lambda: ops.rmsnorm_quant_matmul_batch(y, norm.cpu(), 1e-5, [w]), "swiglu formats": lambda: ops.quant_swiglu(y, w, synth.device_weight("Q5_K", 96, 512, gen)),
        "swiglu shapes": lambda: ops.quant_swiglu(y, w, gate), "mlp shapes": lambda: ops.quant_mlp(y, gate, up, w), "dequantize": lambda: ops.dequantize(w6, torch.bfloat16),
        "dequantize 1-D": lambda: ops.dequantize(flat), "dequantize to int": lambda: ops.dequantize(w, torch.int8), "dequantize on host": lambda: ops.dequantize(on_host)})
    return c


def _outcome(call):
    try:
        r = call()
    except Exception as e:
        return type(e), str(e)
    return [t.clone() for t in (r if isinstance(r, list) else [r])]


def test_both_forms_agree(ops, monkeypatch):
    """The compiled entry points and the Python form of the operators: the same bits, the same refusals in the same words."""
    calls = _calls(ops)
    compiled = {name: _outcome(call) for name, call in calls.items()}
    monkeypatch.setattr(tensor, "_hostops", tensor._PythonForms)
    for name, call in calls.items():
        a, b = compiled[name], _outcome(call)
        assert type(a) is type(b), (name, a, b)
        if isinstance(a, tuple):
            assert a == b, name
        else:
            assert len(a) == len(b) and all(p.shape == q.shape and p.dtype == q.dtype and torch.equal(p, q) for p, q in zip(a, b)), name
    refused = {n for n, r in compiled.items() if isinstance(r, tuple)}
    assert {"half", "K", "out shape", "out type", "outs short", "norm address", "swiglu formats", "mlp shapes", "f64 result"} <= refused
    assert not any(n[-1].isdigit() for n in refused), refused
    ops.check_device_status()


def test_scratch_of_threads_and_streams(ops):
    """Threads on one stream and on their own streams, with scratch that grows on the way: nobody reads another's."""
    gen = _gen(4)
    w = synth.device_weight("Q4_K", 1024, 1024, gen)
    xs = [torch.randn(m, 1024, device="cuda", generator=gen) for m in (5, 600, 20, 12, 300, 40)]
    want = [ops.quant_matmul(x, w) for x in xs]
    torch.cuda.synchronize()
    shared, errors = torch.cuda.Stream(), []

    def work(i):
        try:
            with torch.cuda.stream(shared if i < 4 else torch.cuda.Stream()):
                for r in range(60):
                    j = (i + r) % len(xs)
                    if not torch.equal(ops.quant_matmul(xs[j], w), want[j]):
                        raise AssertionError(f"thread {i}, pass {r}")
        except BaseException as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    ops.check_device_status()


def test_outputs_given_in_part(ops):
    """None among the outputs of a batch: that one is allocated, and returned."""
    gen = _gen(5)
    w = synth.device_weight("Q4_K", 64, 512, gen)
    x = torch.randn(3, 512, device="cuda", generator=gen)
    y = torch.empty(3, 64, device="cuda")
    got = ops.quant_matmul_batch(x, [w, w], outs=[None, y])
    assert got[1] is y and torch.equal(got[0], y) and torch.equal(y, ops.quant_matmul(x, w))
