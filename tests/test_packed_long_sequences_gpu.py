"""Packed sequences of which some are much longer than the others: those run in the 16-row form, the others in the
tensor-memory form.  Every sequence against a call of its own in the form that it should have, to the bit."""
import ctypes

import pytest
import torch

import kda_ascendc_b200 as K
from kda_ascendc_b200 import _lib, api
from oracle import kda_oracle as O
from tests.conftest import to_device

pytestmark = pytest.mark.gpu
FLAGS = dict(use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True, output_final_state=True)


def _long(chunks, H, sms):
    """Which sequences the rule moves: the longest on half of the SMs, above 0.9 x chunks per SM and 1.5 x the mean."""
    n, total = len(chunks), sum(chunks)
    most = min(n - 1, sms // (4 * H))
    if most <= 0 or total * H < 64 * sms:
        return set()
    line = max(9 * total * H // (10 * sms), 3 * total // (2 * n)) + 1
    order = sorted(range(n), key=lambda i: (-chunks[i], i))
    return {i for i in order[:most] if chunks[i] >= line}


def _on_line(rest, H, sms):
    """A first sequence of exactly as many chunks as the rule asks for, in front of `rest` (in chunks)."""
    first = max(rest)
    while 0 not in _long([first] + rest, H, sms):
        first += 1
        assert first < 4000
    return [first] + rest


@pytest.mark.parametrize("H,chunks", [
    (16, [300] + [40] * 9), (8, [20] * 12 + [400, 380, 360, 340, 320, 17]), (8, [5] * 20 + [900, 350]), (32, [3, 320, 30, 5, 2]),
    (16, "at"), (16, "below"), (8, [70] * 20)])
def test_every_sequence_has_the_bits_of_its_form(cuda_device, H, chunks):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if isinstance(chunks, str):
        below = chunks == "below"
        chunks = _on_line([60] * 10, H, sms)
        chunks[0] -= below
        assert (0 in _long(chunks, H, sms)) != below
    lens = [16 * c - (i * 5) % 16 for i, c in enumerate(chunks)]
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    d = to_device(O.make_inputs(1, cu[-1], H, seed0=len(lens), h0_std=None), cuda_device)
    d["g"] = (d["g"].float() - 4.0).bfloat16()     # decays that leave much of the state
    h0 = torch.randn(len(lens), H, 128, 128, device=cuda_device, generator=torch.Generator(cuda_device).manual_seed(5)) * 0.3
    kw = dict(scale=d["scale"], lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"], **FLAGS)
    x = [d[n] for n in ("q", "k", "v", "g", "beta")]
    for _ in range(2):
        o, ht = K.kda_bt16_fwd(*x, initial_state=h0, cu_seqlens=cu, **kw)
    moved = _long(chunks, H, sms)
    for i in range(len(lens)):
        y = [t[:, cu[i]:cu[i + 1]].contiguous() for t in x]
        oi = torch.empty_like(y[2])
        hi = torch.empty(1, H, 128, 128, device=cuda_device)
        ws = torch.empty(K.workspace_bytes(1, lens[i], H), dtype=torch.uint8, device=cuda_device)
        a = api.make_args(*y, scale=d["scale"], lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"], h0=h0[i:i + 1],
                          o=oi, ht=hi, workspace=ws, flags=api._flags(True, True, True), k2_variant=3 if i in moved else 4)
        api._check(_lib.load().kda_fwd(ctypes.byref(a), api._stream_handle()))
        assert api.check_device_status(ws) == 0
        assert torch.equal(o[:, cu[i]:cu[i + 1]], oi) and torch.equal(ht[i:i + 1], hi), (i, chunks[i], i in moved)
