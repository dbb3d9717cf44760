"""The last step of the register forms of K2 is compiled by itself: chains of one chunk up to more chunks than the record ring
has stages, with whole and partial last chunks, in every split, with and without outputs."""
import ctypes

import pytest
import torch

import kda_ascendc_b200 as K
from kda_ascendc_b200 import _lib, api
from oracle import kda_oracle as O
from tests.conftest import to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 16, 17, 32, 47, 64, 65, 80, 81])
@pytest.mark.parametrize("variant,splits", [(1, (4, 8, 16)), (3, (2, 4, 8))])
def test_chain_lengths_around_the_ring(cuda_device, T, variant, splits):
    B, H = 2, 3
    inp = O.make_inputs(B, T, H, seed0=T, h0_std=0.05)
    o_r, ht_r = O.run_chunk_reference(inp)
    d = to_device(inp, cuda_device)
    lib, st = _lib.load(), api._stream_handle()
    ws = torch.empty(K.workspace_bytes(B, T, H), dtype=torch.uint8, device=cuda_device)
    eye = torch.eye(128, device=cuda_device).expand(B, H, 128, 128).contiguous()
    nan = lambda *s, dtype=torch.float32: torch.full(s, float("nan"), dtype=dtype, device=cuda_device)

    def args(vsplit, h0, o, ht):
        return api.make_args(d["q"], d["k"], d["v"], d["g"], d["beta"], scale=d["scale"], lower_bound=d["lower_bound"],
                             A_log=d["A_log"], dt_bias=d["dt_bias"], h0=h0, o=o, ht=ht, workspace=ws, flags=7,
                             k2_variant=variant, k2_vsplit=vsplit)

    def state(vsplit, h0, zero_u, *shape):
        ht = nan(*shape)
        api._check(lib.kda_fwd_k2_state(ctypes.byref(args(vsplit, h0, None, ht)), zero_u, st))
        return ht

    first = None
    for vs in splits:
        o, ht = nan(B, T, H, 128, dtype=torch.bfloat16), nan(B, H, 128, 128)
        a = args(vs, d["initial_state"], o, ht)
        if first is None:
            api._check(lib.kda_fwd_k1(ctypes.byref(a), st))
        api._check(lib.kda_fwd_k2(ctypes.byref(a), st))
        first = first or (o, ht)
        assert torch.equal(o, first[0]) and torch.equal(ht, first[1])
        assert torch.equal(state(vs, d["initial_state"], 0, B, H, 128, 128), ht)
        pair = state(vs, None, 2, B, H, 2, 128, 128)
        assert torch.equal(pair[:, :, 0], state(vs, eye, 1, B, H, 128, 128))
        assert torch.equal(pair[:, :, 1], state(vs, None, 0, B, H, 128, 128))
    assert api.check_device_status(ws) == 0
    # the tolerances of the whole forward on these inputs (tests/test_parity_gpu.py)
    assert (first[0].float().cpu() - o_r.float()).abs().max().item() <= 1e-3
    assert (first[1].cpu() - ht_r).abs().max().item() <= 2e-3
