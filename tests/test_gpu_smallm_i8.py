"""The integer tensor-core small-M kernels (csrc/smallm_i8.cu: Q4_K with 8..16 activation rows, Q8_0 above 16) against the CPU oracle.

The Q4_K kernel takes the matrices with enough 128-row tiles for whole tiles per SM; its integer sums are exact and the f32 block terms are
added in K order: the oracle's BITS.  Q4_K products of 17..63 rows, some of which once were this kernel's, stay in these tests: they are held
to the kernel that takes them now (csrc/kquant_few.cu), with the same bits."""
import os

import numpy as np
import pytest

from boostr_b200 import synth
from boostr_b200.format import QuantFormat as F
from util import describe_mismatch, kq_tile_rows, rel_err, seed_of

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ops():
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    from boostr_b200 import ops as o

    return o


def _qt(w, n, k):
    from boostr_b200.tensor import QuantTensor

    return QuantTensor.from_bytes(w, F.Q4_K, (n, k), device="cuda")


def _threads():
    return os.cpu_count() or 8


# whole tiles per SM: 111 tiles and more on a 148-SM part, 8..16 rows
WHOLE = [(8, 14336, 4096), (16, 14336, 4096), (13, 14250, 2048), (9, 18944, 256), (11, 18800, 1024), (15, 37889, 512), (16, 128256, 4096)]
# above 16 rows: many tiles, few tiles, long K, ragged N, a single row of weights
ABOVE_16 = [(32, 19000, 1024), (17, 128 * 148, 256), (17, 50, 1024), (24, 4096, 14336), (32, 1024, 4096), (20, 4096, 4096), (31, 1, 256), (18, 129, 512),
            (32, 300, 16384)]


@pytest.mark.parametrize("m,n,k", WHOLE)
def test_whole_tiles_have_the_oracles_bits(ops, oracle, m, n, k):
    assert kq_tile_rows("Q4_K", m, n, k) == -1  # not the kernel of kquant_few.cu
    rng = synth.rng_for(91, seed_of(m, n, k))
    act = synth.activations(rng, m, k)
    w = synth.weight_bytes("Q4_K", rng, n, k)
    guard = 4096
    flat = torch.full((2 * guard + m * n,), 777.0, device="cuda")
    got = ops.quant_matmul(torch.from_numpy(act).cuda(), _qt(w, n, k), out=flat[guard:guard + m * n].view(m, n)).cpu().numpy()
    ops.check_device_status()
    assert (flat[:guard] == 777.0).all() and (flat[guard + m * n:] == 777.0).all(), "guard regions were written"
    want = oracle.quant_matmul("Q4_K", act, w, n, threads=_threads())
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), describe_mismatch(got, want)


@pytest.mark.parametrize("m,n,k", ABOVE_16)
def test_q4_k_above_16_rows(ops, oracle, m, n, k):
    rng = synth.rng_for(92, seed_of(m, n, k))
    act = synth.activations(rng, m, k)
    w = synth.weight_bytes("Q4_K", rng, n, k)
    guard = 4096
    flat = torch.full((2 * guard + m * n,), 777.0, device="cuda")
    x = torch.from_numpy(act).cuda()
    qt = _qt(w, n, k)
    got = ops.quant_matmul(x, qt, out=flat[guard:guard + m * n].view(m, n)).cpu().numpy()
    ops.check_device_status()
    assert (flat[:guard] == 777.0).all() and (flat[guard + m * n:] == 777.0).all(), "guard regions were written"
    want = oracle.quant_matmul("Q4_K", act, w, n, threads=_threads())
    e_max, e_rms = rel_err(got, want)
    assert np.isfinite(got).all()
    assert e_max <= 2e-6, f"M={m} N={n} K={k}: {e_max:.3e} (rms {e_rms:.3e})\n" + describe_mismatch(got, want)
    if (n, k) != (300, 16384):  # three tiles of long K: mma.sync, whose chunks of K are added as sums
        assert kq_tile_rows("Q4_K", m, n, k) > 0 and np.array_equal(got.view(np.uint32), want.view(np.uint32)), describe_mismatch(got, want)
    for _ in range(2):
        again = ops.quant_matmul(x, qt).cpu().numpy()
        assert np.array_equal(again.view(np.uint32), got.view(np.uint32))
    ops.check_device_status()


def test_bf16_activations_and_16bit_outputs(ops, oracle):
    m, n, k = 24, 700, 2048
    rng = synth.rng_for(93, 1)
    act = synth.activations(rng, m, k)
    w = synth.weight_bytes("Q4_K", rng, n, k)
    xb = torch.from_numpy(act).cuda().to(torch.bfloat16)
    act_bf = xb.float().cpu().numpy()
    want = oracle.quant_matmul("Q4_K", act_bf, w, n, threads=_threads())
    qt = _qt(w, n, k)
    got = ops.quant_matmul(xb, qt, out_dtype=torch.float32).cpu().numpy()
    assert rel_err(got, want)[0] <= 2e-6
    for dt, tol in ((torch.bfloat16, 2 ** -8), (torch.float16, 2 ** -10)):
        g16 = ops.quant_matmul(xb, qt, out_dtype=dt).float().cpu().numpy()
        assert rel_err(g16, want)[0] <= tol, dt
    ops.check_device_status()


@pytest.mark.parametrize("m,n,k", [(16, 14336, 4096), (32, 512, 1024), (19, 1000, 4096)])
def test_swiglu(ops, oracle, m, n, k):
    rng = synth.rng_for(94, seed_of(m, n, k))
    act = synth.activations(rng, m, k)
    wg = synth.weight_bytes("Q4_K", rng, n, k)
    wu = synth.weight_bytes("Q4_K", rng, n, k)
    got = ops.quant_swiglu(torch.from_numpy(act).cuda(), _qt(wg, n, k), _qt(wu, n, k)).cpu().numpy()
    ops.check_device_status()
    want = oracle.quant_swiglu("Q4_K", act, wg, wu, n, threads=_threads())
    e_max, _ = rel_err(got, want)
    assert e_max <= 1e-5, f"{e_max:.3e}\n" + describe_mismatch(got, want)


def test_zero_rows_and_a_zero_activation_row(ops, oracle):
    # an all-zero activation row quantises with d8 = 0 and must give exact zeros, beside ordinary rows
    m, n, k = 20, 260, 1024
    rng = synth.rng_for(95, 2)
    act = synth.activations(rng, m, k)
    act[7] = 0.0
    w = synth.weight_bytes("Q4_K", rng, n, k)
    got = ops.quant_matmul(torch.from_numpy(act).cuda(), _qt(w, n, k)).cpu().numpy()
    ops.check_device_status()
    want = oracle.quant_matmul("Q4_K", act, w, n, threads=4)
    assert (got[7] == 0.0).all()
    assert rel_err(got, want)[0] <= 2e-6


def test_graph_replay_is_bitwise_identical(ops):
    m, n, k = 32, 2048, 4096
    gen = torch.Generator(device="cuda")
    gen.manual_seed(9)
    w = synth.device_weight("Q4_K", n, k, gen)
    x = torch.randn(m, k, device="cuda", generator=gen)
    y = torch.empty(m, n, device="cuda")
    ref = ops.quant_matmul(x, w).clone()
    for _ in range(2):
        ops.quant_matmul(x, w, out=y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        ops.quant_matmul(x, w, out=y)
    for _ in range(3):
        y.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, ref)
    ops.check_device_status()


# ------------------------------------------------------------------ Q8_0, 17..32 activation rows
# f32 activations on the CPU path; here two int8 pieces per value (relative error ~3e-5 of a 256-run's amax): the bar of
# the small-M kernel above 8 rows, 1e-4 of the largest output.

def _q8(w, n, k):
    from boostr_b200.tensor import QuantTensor

    return QuantTensor.from_bytes(w, F.Q8_0, (n, k), device="cuda")


@pytest.mark.parametrize("m,n,k", [(32, 11008, 4096), (17, 9600, 512), (24, 74 * 128 + 5, 1024), (31, 20000, 256)])
def test_q8_0_above_16_rows(ops, oracle, m, n, k):
    rng = synth.rng_for(96, seed_of(m, n, k))
    act = synth.activations(rng, m, k)
    w = synth.weight_bytes("Q8_0", rng, n, k)
    guard = 4096
    flat = torch.full((2 * guard + m * n,), 555.0, device="cuda")
    x = torch.from_numpy(act).cuda()
    qt = _q8(w, n, k)
    got = ops.quant_matmul(x, qt, out=flat[guard:guard + m * n].view(m, n)).cpu().numpy()
    ops.check_device_status()
    assert (flat[:guard] == 555.0).all() and (flat[guard + m * n:] == 555.0).all(), "guard regions were written"
    want = oracle.quant_matmul("Q8_0", act, w, n, threads=_threads())
    e_max, e_rms = rel_err(got, want)
    assert np.isfinite(got).all()
    assert e_max <= 1e-4, f"M={m} N={n} K={k}: {e_max:.3e} (rms {e_rms:.3e})\n" + describe_mismatch(got, want)
    again = ops.quant_matmul(x, qt).cpu().numpy()
    assert np.array_equal(again.view(np.uint32), got.view(np.uint32))


def test_q8_0_swiglu_and_bf16(ops, oracle):
    m, n, k = 20, 9728, 1024
    rng = synth.rng_for(97, 3)
    act = synth.activations(rng, m, k)
    wg = synth.weight_bytes("Q8_0", rng, n, k)
    wu = synth.weight_bytes("Q8_0", rng, n, k)
    got = ops.quant_swiglu(torch.from_numpy(act).cuda(), _q8(wg, n, k), _q8(wu, n, k)).cpu().numpy()
    ops.check_device_status()
    want = oracle.quant_swiglu("Q8_0", act, wg, wu, n, threads=_threads())
    assert rel_err(got, want)[0] <= 4e-4
    xb = torch.from_numpy(act).cuda().to(torch.bfloat16)
    want_b = oracle.quant_matmul("Q8_0", xb.float().cpu().numpy(), wg, n, threads=_threads())
    got_b = ops.quant_matmul(xb, _q8(wg, n, k)).cpu().numpy()
    assert rel_err(got_b, want_b)[0] <= 1e-4


@pytest.mark.parametrize("fmt,m,n,k", [("Q4_K", 16, 14336, 4096), ("Q4_K", 32, 4096, 4096), ("Q4_K", 24, 4096, 14336), ("Q8_0", 32, 11008, 4096),
                                       ("Q4_K", 17, 1024, 4096)])
def test_many_replays_keep_their_bits_and_never_time_out(ops, fmt, m, n, k):
    # back-to-back launches (the next call's kernels start under programmatic dependent launch while this one drains):
    # every replay must reproduce the first result and no bounded wait may give up
    gen = torch.Generator(device="cuda")
    gen.manual_seed(11)
    ws = [synth.device_weight(fmt, n, k, gen) for _ in range(4)]
    x = torch.randn(m, k, device="cuda", generator=gen)
    y = torch.empty(m, n, device="cuda")
    ref = ops.quant_matmul(x, ws[-1]).clone()

    def run():
        for w in ws:
            ops.quant_matmul(x, w, out=y)

    run()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        run()
    for it in range(100):
        g.replay()
        if it % 20 == 19:
            torch.cuda.synchronize()
            assert torch.equal(y, ref)
    torch.cuda.synchronize()
    ops.check_device_status()


@pytest.mark.parametrize("fmt,m,n,k,tol", [("Q4_K", 40, 14336, 4096, 0.0), ("Q4_K", 63, 700, 1024, 2e-6), ("Q4_K", 33, 19000, 512, 0.0), ("Q8_0", 48, 11008, 1024, 1e-4),
                                           ("Q8_0", 33, 9600, 512, 1e-4)])
def test_33_to_63_rows(ops, oracle, fmt, m, n, k, tol):
    # the bf16 tensor-core path starts at 64 rows; below it Q8_0 goes through the integer kernel in passes of up to 32 rows (a
    # last pass of up to 16 through the mma.sync kernel), Q4_K in one pass through kquant_few.cu
    if fmt == "Q4_K":
        assert kq_tile_rows(fmt, m, n, k) > 0
    from boostr_b200.tensor import QuantTensor

    rng = synth.rng_for(98, seed_of(fmt, m, n, k))
    act = synth.activations(rng, m, k)
    w = synth.weight_bytes(fmt, rng, n, k)
    guard = 4096
    flat = torch.full((2 * guard + m * n,), 333.0, device="cuda")
    qt = QuantTensor.from_bytes(w, F.parse(fmt), (n, k), device="cuda")
    got = ops.quant_matmul(torch.from_numpy(act).cuda(), qt, out=flat[guard:guard + m * n].view(m, n)).cpu().numpy()
    ops.check_device_status()
    assert (flat[:guard] == 333.0).all() and (flat[guard + m * n:] == 333.0).all(), "guard regions were written"
    want = oracle.quant_matmul(fmt, act, w, n, threads=_threads())
    if tol == 0.0:
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), describe_mismatch(got, want)
    else:
        assert rel_err(got, want)[0] <= tol, describe_mismatch(got, want)


@pytest.mark.parametrize("m", [33, 40, 48, 49, 63])
def test_passes_fit_the_scratch_they_ask_for(ops, oracle, m):
    # the last pass may be one of the mma.sync kernel, whose partial sums of a long K need more than the images of 32 rows
    from boostr_b200 import _cabi
    from boostr_b200.tensor import QuantTensor

    n, k, fid = 9600, 8192, F.Q8_0.format_id
    rng = synth.rng_for(99, m)
    act, w = synth.activations(rng, m, k), synth.weight_bytes("Q8_0", rng, n, k)
    qt, x, out = QuantTensor.from_bytes(w, F.Q8_0, (n, k), device="cuda"), torch.from_numpy(act).cuda(), torch.empty(m, n, device="cuda")
    lib = _cabi.lib()
    need = lib.b200q_workspace_bytes(_cabi.OP_QUANT_MATMUL, fid, m, k, n)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    rc = lib.b200q_quant_matmul(fid, x.data_ptr(), _cabi.DT_F32, qt.storage.data_ptr(), out.data_ptr(), _cabi.DT_F32, m, k, n, ws.data_ptr(), need,
                                torch.cuda.current_stream().cuda_stream)
    assert rc == 0, lib.b200q_last_error()
    ops.check_device_status()
    want = oracle.quant_matmul("Q8_0", act, w, n, threads=_threads())
    assert rel_err(out.cpu().numpy(), want)[0] <= 1e-4
