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


def _inputs(B, T, H, g32, flags, dev):
    d = to_device(O.make_inputs(B, T, H, seed0=T, h0_std=0.05), dev)
    if flags == 0:   # a gate that is already the log2 sum over the chunk, at most zero
        d["g"], d["beta"] = -d["g"].float().abs() * 0.1, d["beta"].sigmoid()
    d["g"] = d["g"].float() if g32 else d["g"].bfloat16()
    return d


def _k1(d, flags, lower_bound, debug=False, tables=None):
    """The workspace after K1; debug outputs (and with them the instance in which the flags decide) when asked for."""
    B, T, H = d["v"].shape[:3]
    ws = torch.full((K.workspace_bytes(B, T if tables is None else layout.CHUNK * tables[1], H),), 0xFF, dtype=torch.uint8,
                    device=d["v"].device)
    g_out = torch.empty(B, T, H, 128, device=ws.device) if debug else None
    a = api.make_args(d["q"], d["k"], d["v"], d["g"], d["beta"], scale=d["scale"], lower_bound=lower_bound, A_log=d["A_log"],
                      dt_bias=d["dt_bias"], h0=None, o=None, ht=None, workspace=ws, flags=flags, g_out=g_out)
    if tables is not None:
        a.n_seqs, a.n_chunks = tables[0], tables[1]
        a.chunk_table, a.seq_table = api._ptr(tables[2]), api._ptr(tables[3])
    api._check(_lib.load().kda_fwd_k1(ctypes.byref(a), api._stream_handle()))
    assert api.check_device_status(ws) == 0
    return ws


FORMS = pytest.mark.parametrize("lower_bound,flags", [(-5.0, 7), (-8.0, 7), (-5.0, 0)])
GATES = pytest.mark.parametrize("g32", [False, True])


@FORMS
@GATES
@pytest.mark.parametrize("B,T,H,how", [(1, 1, 1, "dense"), (2, 16, 3, "dense"), (1, 33, 2, "dense"), (3, 1203, 8, "dense"),
                                       (2, 100, 6, "grouped"), (2, 100, 6, "strided")])
def test_forms_write_the_same_records(cuda_device, B, T, H, how, g32, lower_bound, flags):
    d = _inputs(B, T, H, g32, flags, cuda_device)
    if how == "grouped":     # three value heads share a q / k head
        d["q"], d["k"] = d["q"][:, :, ::3].contiguous(), d["k"][:, :, ::3].contiguous()
    elif how == "strided":   # every other head and all but the first token of larger tensors
        for n in ("q", "k", "v", "g", "beta"):
            wide = torch.full((B, T + 1, 2 * H, *d[n].shape[3:]), float("nan"), dtype=d[n].dtype, device=cuda_device)
            wide[:, 1:, ::2] = d[n]
            d[n] = wide[:, 1:, ::2]
    got, want = (_k1(d, flags, lower_bound, debug)[layout.WS_HEADER_BYTES:] for debug in (False, True))
    assert torch.equal(got, want)


@FORMS
@GATES
def test_forms_write_the_same_records_of_packed_sequences(cuda_device, g32, lower_bound, flags):
    """Packed sequences take no debug outputs: each against a call of its own.  Valid rows only: the others of a partial last
    chunk hold what the next sequence's first tokens give, and nothing reads them."""
    cu, H = [0, 1, 17, 49, 348, 1000, 1203], 6
    d = _inputs(1, cu[-1], H, g32, flags, cuda_device)
    ws = _k1(d, flags, lower_bound, tables=api._varlen_tables(cu, cu[-1], H, cuda_device))
    at = 0
    for a, b in zip(cu, cu[1:]):
        want = layout.unpack_records(_k1(dict(d, **{n: d[n][:, a:b] for n in ("q", "k", "v", "g", "beta")}), flags, lower_bound, True),
                                     1, b - a, H)
        got = layout.unpack_records(ws[at:], 1, b - a, H)   # (what stands for its header is not read)
        at += H * ((b - a + 15) // 16) * layout.REC_BYTES
        assert want.keys() == got.keys()
        for n in want:
            assert torch.equal(got[n], want[n]), (n, a, b)
