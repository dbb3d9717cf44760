"""The forward of long sequences, and of about as many chains as SMs, against the CPU oracle, against the 16-row K2, and
against itself through the stage entry points.  These are the shapes that a record of 64 tokens was once written for;
its bounds stay, whatever form runs them.

Bounds: the absolute ones of the 16-token path on benchmark-distributed inputs (o 1e-3, state 2e-3), the reference's
relative 2e-2 of the largest value where states are O(1); against the 16-row K2 one more rounding step of each side
(|o| <= 0.06 has bf16 steps of 2.5e-4)."""
import ctypes

import pytest
import torch

import kda_ascendc_b200 as K
from kda_ascendc_b200 import _lib, api
from oracle import kda_oracle as O
from tests.conftest import to_device

pytestmark = pytest.mark.gpu


def _forward(d, variant=0, cu=None, k_first=False, flags=(True, True, True)):
    h0 = d["initial_state"]
    if k_first and h0 is not None:
        h0 = h0.transpose(-1, -2).contiguous()
    o, ht = api._forward(d["q"], d["k"], d["v"], d["g"], d["beta"], d["scale"], h0, True, *flags, d["lower_bound"],
                         d["A_log"], d["dt_bias"], not k_first, k2_variant=variant, cu_seqlens=cu)
    torch.cuda.synchronize()
    return o, (ht.transpose(-1, -2) if k_first else ht)


def _heads(inp, heads):
    """The oracle's problem for some of the heads."""
    s = dict(inp)
    for n in ("q", "k", "v", "g", "beta"):
        s[n] = inp[n][:, :, heads]
    s["A_log"] = inp["A_log"][heads]
    s["dt_bias"] = inp["dt_bias"].view(-1, 128)[heads].reshape(-1)
    if inp["initial_state"] is not None:
        s["initial_state"] = inp["initial_state"][:, heads]
    return s


# last chunks of 16, 1, 15 and 8 tokens, few and many chains, lower bounds around -5.03, fp32 gates
@pytest.mark.parametrize("B,T,H,lower_bound,g_dtype", [
    (1, 8192, 32, -5.0, torch.bfloat16), (1, 4097, 16, -5.0, torch.float32), (1, 1087, 96, -5.0, torch.bfloat16),
    (4, 1041, 37, -5.0, torch.bfloat16), (1, 3000, 75, -5.02, torch.float32), (1, 3000, 96, -5.04, torch.bfloat16)])
def test_wide_forward_matches_oracle(cuda_device, B, T, H, lower_bound, g_dtype):
    inp = O.make_inputs(B, T, H, seed0=T + H, h0_std=0.05, g_dtype=g_dtype)
    inp["lower_bound"] = lower_bound
    d = to_device(inp, cuda_device)
    o, ht = _forward(d)
    heads = [0, H // 2, H - 1]
    o_r, ht_r = O.run_chunk_reference(_heads(inp, heads))
    assert (o[:, :, heads].float().cpu() - o_r.float()).abs().max().item() <= 1e-3
    assert (ht[:, heads].cpu() - ht_r).abs().max().item() <= 2e-3
    o3, ht3 = _forward(d, variant=3)
    assert (o.float() - o3.float()).abs().max().item() <= 7.5e-4
    assert (ht - ht3).abs().max().item() <= 2e-4
    ok, htk = _forward(d, k_first=True)
    assert torch.equal(o, ok) and torch.equal(ht, htk)


# states that persist: every hand-over between chunks shows
@pytest.mark.parametrize("B,T,H,regime", [(1, 16384, 16, "carry"), (1, 16421, 13, "carry"), (2, 2100, 60, "carry"),
                                          (1, 8200, 32, "long_memory"), (1, 4100, 1, "carry")])
def test_wide_forward_carries_the_state(cuda_device, B, T, H, regime):
    inp = O.make_inputs(B, T, H, seed0=7, regime=regime, h0_std=0.3)
    o, ht = _forward(to_device(inp, cuda_device))
    heads = sorted({H // 2, H - 1})
    o_r, ht_r = O.run_chunk_reference(_heads(inp, heads))
    assert (o[:, :, heads].float().cpu() - o_r.float()).abs().max().item() <= 2e-2 * o_r.float().abs().max().item()
    assert (ht[:, heads].cpu() - ht_r).abs().max().item() <= 2e-2 * ht_r.abs().max().item()


def _stage_args(d, B, T, H, dev, **kw):
    o = torch.full((B, T, H, 128), float("nan"), dtype=torch.bfloat16, device=dev)
    ht = torch.full((B, H, 128, 128), float("nan"), device=dev)
    ws = torch.full((K.workspace_bytes(B, T, H),), 0xFF, dtype=torch.uint8, device=dev)
    a = api.make_args(d["q"], d["k"], d["v"], d["g"], d["beta"], scale=d["scale"], lower_bound=d["lower_bound"],
                      A_log=d["A_log"], dt_bias=d["dt_bias"], h0=d["initial_state"], o=o, ht=ht, workspace=ws,
                      flags=api._flags(True, True, True), **kw)
    return a, o, ht, ws


@pytest.mark.parametrize("B,T,H", [(1, 8192, 32), (2, 1500, 60), (1, 40000, 8)])
def test_stages_equal_the_whole_forward(cuda_device, B, T, H):
    """kda_fwd_k1 + kda_fwd_k2 = kda_fwd, o over v = o beside it, and a captured forward follows its inputs: the same bits.
    The state passes over the same records: h0 -> ht, and M, Q with h0 M + Q = ht."""
    d = to_device(O.make_inputs(B, T, H, seed0=3, regime="carry", h0_std=0.3), cuda_device)
    lib, st = _lib.load(), api._stream_handle()
    a, o, ht, ws = _stage_args(d, B, T, H, cuda_device)
    api._check(lib.kda_fwd(ctypes.byref(a), st))
    assert api.check_device_status(ws) == 0
    b, o2, ht2, ws2 = _stage_args(d, B, T, H, cuda_device)
    api._check(lib.kda_fwd_k1(ctypes.byref(b), st))
    api._check(lib.kda_fwd_k2(ctypes.byref(b), st))
    assert api.check_device_status(ws2) == 0 and torch.equal(o, o2) and torch.equal(ht, ht2)
    api._check(lib.kda_fwd_k1(ctypes.byref(b), st))
    api._check(lib.kda_fwd_k2_state(ctypes.byref(b), 0, st))
    top = ht.abs().max().item()
    assert (ht2 - ht).abs().max().item() <= 1e-2 * top
    mq = torch.empty(B * H, 2, 128, 128, device=cuda_device)
    b.ht = mq.data_ptr()
    api._check(lib.kda_fwd_k2_state(ctypes.byref(b), 2, st))
    assert api.check_device_status(ws2) == 0
    walked = d["initial_state"].view(-1, 128, 128).double() @ mq[:, 0].double() + mq[:, 1].double()
    assert (walked - ht.view(-1, 128, 128)).abs().max().item() <= 1e-2 * top
    v = d["v"].clone()
    c, _, ht3, ws3 = _stage_args(dict(d, v=v), B, T, H, cuda_device)
    c.o = v.data_ptr()
    api._check(lib.kda_fwd(ctypes.byref(c), st))
    assert api.check_device_status(ws3) == 0 and torch.equal(v, o) and torch.equal(ht3, ht)
    plan = K.ForwardPlan(d["q"], d["k"], d["v"], d["g"], d["beta"], scale=d["scale"], initial_state=d["initial_state"],
                         lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"])
    plan.run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.run()
    d["v"].mul_(-0.5)
    graph.replay()
    got = plan.o.clone(), plan.final_state.clone()
    o4, ht4 = _forward(d)
    assert torch.equal(got[0], o4) and torch.equal(got[1], ht4)


def test_workspace_that_was_sized_for_16_token_records_is_enough(cuda_device):
    """Nothing is written behind kda_fwd_workspace_bytes."""
    for B, T, H in ((1, 8192, 32), (1, 40000, 8), (2, 1500, 60)):
        d = to_device(O.make_inputs(B, T, H, seed0=3, h0_std=0.05), cuda_device)
        a, o, ht, ws = _stage_args(d, B, T, H, cuda_device)     # o and ht live on: a freed o could become `guarded`
        n = ws.numel()
        guarded = torch.full((n + 4096,), 0x5A, dtype=torch.uint8, device=cuda_device)
        a.workspace = guarded.data_ptr()
        api._check(_lib.load().kda_fwd(ctypes.byref(a), api._stream_handle()))
        torch.cuda.synchronize()
        assert bool((guarded[n:] == 0x5A).all()) and int(guarded[:4].view(torch.int32)) == 0
