"""The forward whose K2 runs beside its K1 against the same two kernels one after the other: the same bits."""
import ctypes
import subprocess
import sys
from pathlib import Path

import pytest
import torch

import kda_ascendc_b200 as K
from kda_ascendc_b200 import _lib, api
from oracle import kda_oracle as O
from tests.conftest import to_device

pytestmark = pytest.mark.gpu


def _args(d, o, ht, ws, prepared=False, flags=None, g_out=None):
    if flags is None:
        flags = 0 if prepared else api._flags(True, True, True)
    return api.make_args(d["q"], d["k"], d["v"], d["g"], d["beta"], scale=d["scale"], lower_bound=d["lower_bound"],
                         A_log=d["A_log"], dt_bias=d["dt_bias"], h0=d["initial_state"], o=o, ht=ht, workspace=ws,
                         flags=flags, g_out=g_out)


def _buffers(B, T, H, dev):
    return (torch.full((B, T, H, 128), float("nan"), dtype=torch.bfloat16, device=dev),
            torch.full((B, H, 128, 128), float("nan"), dtype=torch.float32, device=dev),
            torch.full((K.workspace_bytes(B, T, H),), 0xFF, dtype=torch.uint8, device=dev))


def _after(d, B, T, H, dev, **kw):
    o, ht, ws = _buffers(B, T, H, dev)
    a, lib, st = _args(d, o, ht, ws, **kw), _lib.load(), api._stream_handle()
    api._check(lib.kda_fwd_k1(ctypes.byref(a), st))
    api._check(lib.kda_fwd_k2(ctypes.byref(a), st))
    assert api.check_device_status(ws) == 0
    return o, ht


def _whole(d, B, T, H, dev, launches=None, **kw):
    o, ht, ws = _buffers(B, T, H, dev)
    a = _args(d, o, ht, ws, **kw)
    api._check(_lib.load().kda_fwd(ctypes.byref(a), api._stream_handle()))
    if launches is not None and _sms() == 148:   # the lines between the forms are in SMs
        assert _lib.load().kda_last_launch_count() == launches
    assert api.check_device_status(ws) == 0
    return o, ht


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


AFTER, BESIDE = 2, 3   # launches of a forward: K1 and K2, and beside K1 the kernel that clears the header


# 8-row form (chains x 8 <= SMs) and tensor-memory form (up to 13/14 of the SMs), on both sides of the
# rule's line of 16 items per SM and of its line in chains; whole and partial last windows and chunks
@pytest.mark.parametrize("B,T,H,lower_bound,prepared,launches", [
    (1, 4736, 8, -5.0, False, BESIDE), (1, 4720, 8, -5.0, False, AFTER), (2, 2353, 8, -5.0, False, BESIDE),
    (1, 40001, 1, -5.0, False, BESIDE), (3, 9000, 6, -5.0, False, BESIDE), (2, 2400, 8, -8.0, False, BESIDE),
    (2, 2400, 8, -5.0, True, BESIDE), (1, 16 * 121 + 5, 18, -5.0, False, AFTER), (1, 531, 75, -5.0, False, BESIDE),
    (1, 1024, 96, -5.0, False, BESIDE), (3, 1003, 37, -5.0, False, BESIDE), (1, 530, 112, -5.0, False, BESIDE),
    (1, 20, 96, -5.0, False, AFTER)])
def test_beside_equals_after(cuda_device, B, T, H, lower_bound, prepared, launches):
    d = to_device(O.make_inputs(B, T, H, seed0=T + H, h0_std=0.05), cuda_device)
    d["lower_bound"] = lower_bound
    if prepared:   # what a caller that normalises and sums the gate itself hands over
        d["q"], d["k"] = (torch.nn.functional.normalize(d[n].float(), dim=-1).bfloat16() for n in ("q", "k"))
        d["g"] = -d["g"].float().abs() * 0.1
        d["beta"] = d["beta"].sigmoid()
    ref = _after(d, B, T, H, cuda_device, prepared=prepared)
    for _ in range(3):
        got = _whole(d, B, T, H, cuda_device, launches, prepared=prepared)
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])


# K2 on SMs of its own: the 8-row form with four consumer warps, the 16-row form in place of the 8-row one and as chosen, the
# tensor-memory form with two CTAs per SM and with one; both sides of the lines between them, partial last chunks.  Decays
# that leave much of the state, so that every step matters to the last bit.
@pytest.mark.parametrize("B,T,H,launches", [
    (1, 1991, 19, BESIDE), (1, 1570, 24, BESIDE), (1, 1616, 32, AFTER), (1, 1630, 32, BESIDE), (1, 1157, 37, BESIDE),
    (2, 1531, 19, BESIDE), (1, 1530, 42, BESIDE), (1, 1521, 43, AFTER), (1, 4085, 80, BESIDE), (1, 4085, 81, BESIDE),
    (1, 4067, 103, BESIDE), (1, 4090, 103, BESIDE), (1, 1500, 104, BESIDE), (1, 531, 137, BESIDE), (1, 531, 138, AFTER)])
def test_beside_equals_after_where_k2_has_sms_of_its_own(cuda_device, B, T, H, launches):
    d = to_device(O.make_inputs(B, T, H, seed0=T + H, h0_std=0.3), cuda_device)
    d["g"] = (d["g"].float() - 4.0).bfloat16()
    ref = _after(d, B, T, H, cuda_device)
    for _ in range(2):
        got = _whole(d, B, T, H, cuda_device, launches)
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])


# the 8-row, the 16-row (in place of the 8-row and as chosen) and the tensor-memory form on SMs of their own
@pytest.mark.parametrize("B,T,H", [(1, 1991, 19), (1, 1630, 32), (2, 1531, 19), (1, 4085, 81)])
@pytest.mark.parametrize("g32,k_first", [(True, False), (False, True), (True, True)])
def test_either_gate_type_and_state_order_where_k2_has_sms_of_its_own(cuda_device, B, T, H, g32, k_first):
    d = to_device(O.make_inputs(B, T, H, seed0=T + H, h0_std=0.3), cuda_device)
    d["g"] = (d["g"].float() - 4.0).to(torch.float32 if g32 else torch.bfloat16)
    flags = api._flags(True, True, True) | (_lib.FLAG_STATE_K_FIRST if k_first else 0)
    ref = _after(d, B, T, H, cuda_device, flags=flags)
    got = _whole(d, B, T, H, cuda_device, BESIDE, flags=flags)
    assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])


# one chunk, fewer chunks than stages of the record ring, more; a partial last chunk
@pytest.mark.parametrize("T", [5, 16, 33, 64, 100, 1003])
@pytest.mark.parametrize("k_first", [False, True])
def test_both_register_forms_give_the_same_bits(cuda_device, T, k_first):
    B, H = 2, 3
    d = to_device(O.make_inputs(B, T, H, seed0=T, h0_std=0.3), cuda_device)
    d["g"] = (d["g"].float() - 4.0).bfloat16()
    flags = api._flags(True, True, True) | (_lib.FLAG_STATE_K_FIRST if k_first else 0)
    lib, st, got = _lib.load(), api._stream_handle(), []
    for variant, splits in ((1, (4, 8, 16)), (3, (2, 4, 8))):
        for vsplit in splits:
            o, ht, ws = _buffers(B, T, H, cuda_device)
            a = _args(d, o, ht, ws, flags=flags)
            a.k2_variant, a.k2_vsplit = variant, vsplit
            api._check(lib.kda_fwd(ctypes.byref(a), st))
            assert api.check_device_status(ws) == 0
            got.append((o, ht))
    for o, ht in got[1:]:
        assert torch.equal(o, got[0][0]) and torch.equal(ht, got[0][1])


# K1 beside K2 is compiled for either gate type and centring, with all three of gate, l2-norm and sigmoid in the kernel, with
# none of them (general centring only), and with the flags deciding (some of them, or debug outputs): all ten instances, in
# front of either form of K2
@pytest.mark.parametrize("B,T,H", [(2, 2400, 8), (1, 531, 75)])
@pytest.mark.parametrize("g32", [False, True])
@pytest.mark.parametrize("flags,lower_bound,debug", [(7, -5.0, False), (7, -8.0, False), (0, -5.0, False), (2, -5.0, False),
                                                     (5, -5.0, False), (5, -8.0, False), (7, -5.0, True), (7, -8.0, True)])
def test_beside_equals_after_in_every_instance_of_k1(cuda_device, B, T, H, g32, flags, lower_bound, debug):
    d = to_device(O.make_inputs(B, T, H, seed0=T + H, h0_std=0.05), cuda_device)
    d["lower_bound"] = lower_bound
    if not flags & _lib.FLAG_GATE:
        d["g"] = -d["g"].float().abs() * 0.1
    if not flags & _lib.FLAG_L2NORM:
        d["q"], d["k"] = (torch.nn.functional.normalize(d[n].float(), dim=-1).bfloat16() for n in ("q", "k"))
    if not flags & _lib.FLAG_BETA_SIGMOID:
        d["beta"] = d["beta"].sigmoid()
    d["g"] = d["g"].float() if g32 else d["g"].bfloat16()
    g_out = [torch.full((B, T, H, 128), float("nan"), device=cuda_device) if debug else None for _ in range(2)]
    ref = _after(d, B, T, H, cuda_device, flags=flags, g_out=g_out[0])
    got = _whole(d, B, T, H, cuda_device, flags=flags, g_out=g_out[1])
    assert got[0].isfinite().all() and got[1].isfinite().all()
    assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
    assert not debug or torch.equal(g_out[0], g_out[1])


def test_output_over_an_input(cuda_device):
    """o over v: K2 may not write outputs before K1 has read the values."""
    B, T, H = 2, 2400, 8
    d = to_device(O.make_inputs(B, T, H, seed0=5, h0_std=0.05), cuda_device)
    ref = _after(d, B, T, H, cuda_device)
    _, ht, ws = _buffers(B, T, H, cuda_device)
    a = _args(d, d["v"], ht, ws)
    api._check(_lib.load().kda_fwd(ctypes.byref(a), api._stream_handle()))
    assert torch.equal(d["v"], ref[0]) and torch.equal(ht, ref[1])


@pytest.mark.parametrize("B,T,H", [(2, 2400, 8), (1, 600, 96), (1, 100, 32)])
def test_captured_forward_follows_its_inputs(cuda_device, B, T, H):
    """Both kernels in a CUDA graph, replayed back to back on changing inputs."""
    d = to_device(O.make_inputs(B, T, H, seed0=9, h0_std=0.05), cuda_device)
    plan = K.ForwardPlan(d["q"], d["k"], d["v"], d["g"], d["beta"], scale=d["scale"], initial_state=d["initial_state"],
                         lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"])
    plan.run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.run()
    for _ in range(3):
        d["v"].mul_(-0.5)
        graph.replay()
        got = plan.o.clone(), plan.final_state.clone()
        ref = _after(d, B, T, H, cuda_device)
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])


# the 8-row and the 16-row form (full barrier: 2) and the tensor-memory form (any of its waits: 4)
@pytest.mark.parametrize("B,T,H,own", [(1, 4736, 8, 2), (1, 600, 96, 4), (1, 1991, 19, 2), (1, 1630, 32, 2), (1, 1530, 42, 2)])
@pytest.mark.parametrize("k1_status", [0, 1])
def test_window_wait_runs_out(cuda_device, B, T, H, own, k1_status):
    """K2 on window counters that nothing counts up: it gives up after its limit, the outputs are left alone and the
    next forward works.  After a K1 that gave up (its word of the header), that is what the status names."""
    d = to_device(O.make_inputs(B, T, H, seed0=11, h0_std=0.05), cuda_device)
    o, ht, ws = _buffers(B, T, H, cuda_device)
    header = ws[:8].view(torch.int32)
    header.copy_(torch.tensor([0, k1_status]))
    a = _args(d, o, ht, ws)
    api._check(_lib.load().kda_selftest_window_wait(ctypes.byref(a), api._stream_handle()))
    torch.cuda.synchronize()
    assert int(header[0]) in (8, own) and int(header[1]) == k1_status
    assert o.isnan().all() and ht.isnan().all()
    status = ctypes.c_int32(-1)
    assert _lib.load().kda_fwd_status(api._ptr(ws), api._stream_handle(), ctypes.byref(status)) == -3
    assert status.value == (k1_status or int(header[0]))
    api._check(_lib.load().kda_fwd(ctypes.byref(a), api._stream_handle()))
    assert api.check_device_status(ws) == 0
    ref = _after(d, B, T, H, cuda_device)
    assert torch.equal(o, ref[0]) and torch.equal(ht, ref[1])


def test_k1_clears_both_status_words(cuda_device):
    B, T, H = 1, 100, 3
    d = to_device(O.make_inputs(B, T, H, seed0=11, h0_std=0.05), cuda_device)
    o, ht, ws = _buffers(B, T, H, cuda_device)
    a = _args(d, o, ht, ws)
    api._check(_lib.load().kda_fwd_k1(ctypes.byref(a), api._stream_handle()))
    assert ws[:8].view(torch.int32).tolist() == [0, 0]


def test_window_wait_selftest_refuses_other_forwards(cuda_device):
    d = to_device(O.make_inputs(1, 100, 32, seed0=11, h0_std=0.05), cuda_device)
    a = _args(d, *_buffers(1, 100, 32, cuda_device))
    assert _lib.load().kda_selftest_window_wait(ctypes.byref(a), api._stream_handle()) == -1
    assert "beside" in _lib.last_error()


def test_first_use_from_several_threads():
    """The first calls of a process, from eight threads at once on streams of their own: what a launch looks up once per
    device must be complete when another thread sees it."""
    body = """
import threading, torch
import kda_ascendc_b200 as K
from oracle import kda_oracle as O
from tests.conftest import to_device
dev = torch.device("cuda:0")
d = [to_device(O.make_inputs(B, T, H, seed0=7, h0_std=0.05), dev) for B, T, H in ((2, 2400, 8), (1, 600, 96)) * 4]
plans = [K.ForwardPlan(x["q"], x["k"], x["v"], x["g"], x["beta"], scale=x["scale"], initial_state=x["initial_state"],
                       lower_bound=x["lower_bound"], A_log=x["A_log"], dt_bias=x["dt_bias"]) for x in d]
streams = [torch.cuda.Stream() for _ in plans]
torch.cuda.synchronize()
start, errors = threading.Barrier(len(plans)), []
def work(i):
    try:
        start.wait()
        plans[i].run(streams[i].cuda_stream)
    except Exception as e:
        errors.append(repr(e))
threads = [threading.Thread(target=work, args=(i,)) for i in range(len(plans))]
[t.start() for t in threads]
[t.join() for t in threads]
torch.cuda.synchronize()
assert not errors, errors
got = [(p.o.clone(), p.final_state.clone()) for p in plans]
for p, (o, ht) in zip(plans, got):
    p.run()
    assert torch.equal(p.o, o) and torch.equal(p.final_state, ht)
"""
    r = subprocess.run([sys.executable, "-c", body], cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
