"""The native host path (csrc/kda_host.cpp) launches what the Python path launches: bit-equal results for the
options that change its argument block, and refusals that end in the Python path's own errors."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

import kda_ascendc_b200 as K
from conftest import to_device
from kda_ascendc_b200 import _lib, api, fla_backend
from oracle import kda_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,v_first,g_dtype,cu", [
    (1, 1, 1, True, torch.bfloat16, None), (2, 33, 3, False, torch.float32, None),
    (1, 70, 2, True, torch.bfloat16, [0, 1, 33, 70]), (1, 70, 2, False, torch.float32, torch.tensor([0, 16, 70])),
    (1, 70, 2, True, torch.bfloat16, torch.tensor([0, 69, 70], dtype=torch.int32, device="meta"))])
def test_chunk_call_equals_the_python_path(cuda_device, B, T, H, v_first, g_dtype, cu):
    d = to_device(O.make_inputs(B, T, H, seed0=3, h0_std=0.1, g_dtype=g_dtype), cuda_device)
    if torch.is_tensor(cu) and cu.is_meta:      # offsets that live on the GPU
        cu = torch.tensor([0, 69, 70], dtype=torch.int32, device=cuda_device)
    if cu is not None:
        d["initial_state"] = d["initial_state"].expand(len(cu) - 1, H, 128, 128).contiguous()
    args = (d["q"], d["k"], d["v"], d["g"], d["beta"])
    want = api._forward(*args, d["scale"], d["initial_state"], True, True, True, True, d["lower_bound"], d["A_log"],
                        d["dt_bias"], v_first, cu_seqlens=cu)
    native = _lib.host().chunk(*args, d["scale"], d["initial_state"], True, True, True, True, True, d["lower_bound"],
                               d["A_log"], d["dt_bias"], v_first, cu, False)
    assert torch.equal(native[0], want[0]) and torch.equal(native[1], want[1])
    # what the native path does not take (here: a numpy scale) is served by the Python path
    kw = dict(initial_state=d["initial_state"], output_final_state=True, use_qk_l2norm_in_kernel=True,
              use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True, lower_bound=d["lower_bound"], A_log=d["A_log"],
              dt_bias=d["dt_bias"], state_v_first=v_first, cu_seqlens=cu)
    o, ht = K.kda_bt16_fwd(*args, scale=np.float64(d["scale"]), **kw)
    assert torch.equal(o, want[0]) and torch.equal(ht, want[1])
    with pytest.raises(ValueError, match="initial_state.shape"):
        K.kda_bt16_fwd(*args, **dict(kw, initial_state=d["initial_state"][:, :, :64].contiguous()))


@pytest.mark.parametrize("T,inplace", [(1, False), (1, True), (api.RECURRENT_MAX_TOKENS + 1, True)])
def test_recurrent_call_takes_strided_views(cuda_device, T, inplace):
    d = to_device(O.make_inputs(2, 2 * T, 3, seed0=4, h0_std=0.1), cuda_device)
    args = tuple(d[n][:, :T] for n in ("q", "k", "v", "g", "beta"))          # batch stride of 2 T tokens
    kw = dict(lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"])
    want = K.kda_recurrent_fwd(*(a.contiguous() for a in args), initial_state=d["initial_state"], **kw)
    st = d["initial_state"].clone()
    o, ht = K.kda_recurrent_fwd(*args, initial_state=st, inplace_state=inplace, **kw)
    assert torch.equal(o, want[0]) and torch.equal(ht, want[1]) and (ht is st) == inplace


def test_out_of_memory_keeps_its_type(cuda_device):
    d = to_device(O.make_inputs(1, 1, 32, seed0=5, h0_std=None), cuda_device)
    args = tuple(d[n].expand(2048, *d[n].shape[1:]).contiguous() for n in ("q", "k", "v", "g", "beta"))
    kw = dict(lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"])
    torch.cuda.empty_cache()
    torch.cuda.set_per_process_memory_fraction(0.02)     # 3.6 GB of 180; the returned state alone takes 4.3
    try:
        with pytest.raises(torch.OutOfMemoryError):
            K.kda_recurrent_fwd(*args, **kw)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    o, ht = K.kda_recurrent_fwd(*(a[:2] for a in args), **kw)
    assert torch.equal(o[0], o[1]) and torch.equal(ht[0], ht[1]) and ht.abs().sum().item() > 0


def _chunk_kw(d):
    return dict(initial_state=d["initial_state"], output_final_state=True, use_qk_l2norm_in_kernel=True,
                use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True, lower_bound=d["lower_bound"], A_log=d["A_log"])


def test_calls_follow_the_current_stream(cuda_device):
    d = to_device(O.make_inputs(1, 100, 4, seed0=6, h0_std=0.1), cuda_device)
    rest = (d["g"], d["beta"])
    rec = dict(lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"], initial_state=d["initial_state"])
    v2 = d["v"] * -0.5
    want = K.kda_bt16_fwd(d["q"], d["k"], v2, *rest, dt_bias=d["dt_bias"], **_chunk_kw(d))
    one = lambda v: tuple(x[:, :1] for x in (d["q"], d["k"], v, *rest))
    want1 = K.kda_recurrent_fwd(*one(v2), **rec)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)            # about 10 ms: a launch on another stream would read v unchanged
        d["v"].mul_(-0.5)
        got = K.kda_bt16_fwd(d["q"], d["k"], d["v"], *rest, dt_bias=d["dt_bias"], **_chunk_kw(d))
        got1 = K.kda_recurrent_fwd(*one(d["v"]), **rec)
    side.synchronize()
    for a, b in zip((*got, *got1), (*want, *want1)):
        assert torch.equal(a, b)


def test_adapter_takes_the_bias_per_head(cuda_device):
    d = to_device(O.make_inputs(1, 50, 4, seed0=7, h0_std=0.1), cuda_device)
    args, kw = (d["q"], d["k"], d["v"], d["g"], d["beta"]), _chunk_kw(d)
    bias = d["dt_bias"].view(4, 128)
    assert bias.abs().max().item() > 0
    want = K.kda_bt16_fwd(*args, dt_bias=d["dt_bias"], scale=d["scale"], **kw)
    got = fla_backend.chunk_kda(*args, dt_bias=bias, scale=d["scale"], safe_gate=True, transpose_state_layout=True, **kw)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    one = tuple(a[:, :1] for a in args)
    want = K.kda_recurrent_fwd(*one, initial_state=d["initial_state"], lower_bound=d["lower_bound"], A_log=d["A_log"],
                               dt_bias=d["dt_bias"], scale=d["scale"])
    got = fla_backend.fused_recurrent_kda(*one, dt_bias=bias, scale=d["scale"], transpose_state_layout=True, **kw)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_offsets_on_the_gpu_under_capture_are_an_ordinary_error():
    """Reading them back is not allowed while the stream is captured; the process goes on."""
    body = """
import torch
import kda_ascendc_b200 as K
from oracle import kda_oracle as O
from tests.conftest import to_device
d = to_device(O.make_inputs(1, 40, 2, seed0=8, h0_std=None), torch.device("cuda:0"))
cu = torch.tensor([0, 17, 40], dtype=torch.int32, device="cuda:0")
call = lambda: K.kda_bt16_fwd(d["q"], d["k"], d["v"], d["g"], d["beta"], cu_seqlens=cu, output_final_state=True,
                              use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True,
                              lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"])
want = call()
torch.cuda.synchronize()
try:
    with torch.cuda.graph(torch.cuda.CUDAGraph()):
        call()
except RuntimeError as e:
    assert "captur" in str(e), e
else:
    raise SystemExit("no error")
got = call()
torch.cuda.synchronize()
assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
"""
    r = subprocess.run([sys.executable, "-c", body], cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]


def test_long_recurrent_call_shares_no_scratch(cuda_device):
    """A call that takes the Python path and the chunk kernels: calls of one shape on two streams may overlap."""
    T = api.RECURRENT_MAX_TOKENS + 1
    d = to_device(O.make_inputs(1, T, 3, seed0=9, h0_std=0.1), cuda_device)
    args = tuple(d[n] for n in ("q", "k", "v", "g", "beta"))
    kw = dict(lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"], initial_state=d["initial_state"])
    kept = dict(api._WORKSPACE_CACHE)
    o, ht = K.kda_recurrent_fwd(*args, scale=np.float64(d["scale"]), **kw)
    assert api._WORKSPACE_CACHE.keys() == kept.keys()
    want = K.kda_recurrent_fwd(*args, scale=d["scale"], **kw)
    assert torch.equal(o, want[0]) and torch.equal(ht, want[1])
