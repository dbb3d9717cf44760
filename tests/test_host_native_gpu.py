"""The native host path (csrc/kda_host.cpp) launches what the Python path launches: bit-equal results for the
options that change its argument block, and refusals that end in the Python path's own errors."""
import numpy as np
import pytest
import torch

import kda_ascendc_b200 as K
from conftest import to_device
from kda_ascendc_b200 import _lib, api
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
