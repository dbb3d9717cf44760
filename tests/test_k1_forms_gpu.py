"""K1 in the instances for calls whose flags are known when it is compiled, against the instance in which the flags decide
(the one that writes the debug outputs): the same records, to the bit."""
import ctypes

import pytest
import torch

import kda_ascendc_b200 as K
from kda_ascendc_b200 import _lib, api, layout
from oracle import kda_oracle as O
from tests.conftest import to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lower_bound,flags", [(-5.0, 7), (-8.0, 7), (-5.0, 0)])
@pytest.mark.parametrize("g32", [False, True])
@pytest.mark.parametrize("B,T,H", [(1, 1, 1), (2, 16, 3), (1, 33, 2), (3, 1203, 8)])
def test_forms_write_the_same_records(cuda_device, B, T, H, g32, lower_bound, flags):
    d = to_device(O.make_inputs(B, T, H, seed0=T, h0_std=0.05), cuda_device)
    g, beta = d["g"], d["beta"]
    if flags == 0:   # a gate that is already the log2 sum over the chunk, at most zero
        g, beta = -g.float().abs() * 0.1, beta.sigmoid()
    g = g.float() if g32 else g.bfloat16()
    got = []
    for debug in (False, True):
        ws = torch.full((K.workspace_bytes(B, T, H),), 0xFF, dtype=torch.uint8, device=cuda_device)
        g_out = torch.empty(B, T, H, 128, device=cuda_device) if debug else None
        a = api.make_args(d["q"], d["k"], d["v"], g, beta, scale=d["scale"], lower_bound=lower_bound, A_log=d["A_log"],
                          dt_bias=d["dt_bias"], h0=None, o=None, ht=None, workspace=ws, flags=flags, g_out=g_out)
        api._check(_lib.load().kda_fwd_k1(ctypes.byref(a), api._stream_handle()))
        assert api.check_device_status(ws) == 0
        got.append(ws[layout.WS_HEADER_BYTES:].clone())
    assert torch.equal(got[0], got[1])
