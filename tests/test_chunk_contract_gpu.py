"""What the forward promises about its chunks of 16 tokens at the sizes that production calls have: a sequence may be cut
at any chunk boundary, a stage call takes the records of any earlier K1, and a token that is not finite reaches back no
further than its own chunk.  All comparisons are of bits: both sides run the same kernels on the same records."""
import ctypes

import pytest
import torch

import kda_ascendc_b200 as K
from kda_ascendc_b200 import _lib, api

pytestmark = pytest.mark.gpu
D = 128
UNSUPPORTED = -4          # KDA_ERR_UNSUPPORTED


def _inputs(dev, B, T, H, seed):
    g = torch.Generator(device=dev).manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)
    return dict(q=rn(B, T, H, D).bfloat16(), k=rn(B, T, H, D).bfloat16(), v=rn(B, T, H, D).bfloat16(),
                g=(rn(B, T, H, D) - 4.0).bfloat16(), beta=rn(B, T, H),       # decays that leave much of the state
                A_log=torch.zeros(H, device=dev), dt_bias=torch.rand(H * D, device=dev, generator=g) * 0.2 - 0.1,
                h0=rn(B, H, D, D) * 0.3)


def _fwd(d, a=0, b=None, h0=None):
    x = [d[n][:, a:b].contiguous() for n in ("q", "k", "v", "g", "beta")]
    return K.kda_bt16_fwd(*x, scale=D ** -0.5, initial_state=d["h0"] if h0 is None else h0, output_final_state=True,
                          use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True,
                          lower_bound=-5.0, A_log=d["A_log"], dt_bias=d["dt_bias"])


class _Call:
    """An argument block with buffers of its own, filled with what no kernel writes."""

    def __init__(self, d, **kw):
        B, T, H = d["beta"].shape
        dev = d["q"].device
        self.o = torch.full((B, T, H, D), float("nan"), dtype=torch.bfloat16, device=dev)
        self.ht = torch.full((B, H, D, D), float("nan"), device=dev)
        self.ws = torch.full((K.workspace_bytes(B, T, H),), 0xFF, dtype=torch.uint8, device=dev)
        self.args = api.make_args(d["q"], d["k"], d["v"], d["g"], d["beta"], scale=D ** -0.5, lower_bound=-5.0,
                                  A_log=d["A_log"], dt_bias=d["dt_bias"], h0=d["h0"], o=self.o, ht=self.ht,
                                  workspace=self.ws, flags=api._flags(True, True, True), **kw)

    def __call__(self, name, *more):
        api._check(getattr(_lib.load(), name)(ctypes.byref(self.args), *more, api._stream_handle()))
        return self

    def result(self):
        assert api.check_device_status(self.ws) == 0
        return self.o, self.ht


def _same(a, b):
    return torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


# cuts that are multiples of 16 only, of 32, of 64; 8-row and tensor-memory K2; beside K1 and after it
@pytest.mark.parametrize("B,T,H,cut", [
    (1, 8192, 32, 4112), (2, 4096, 8, 2064), (1, 4096, 16, 4064), (1, 16384, 16, 1040), (1, 8192, 96, 4112),
    (1, 3000, 75, 2400), (1, 3000, 148, 1024), (3, 2000, 48, 1488)])
def test_continuation_at_any_chunk_boundary(cuda_device, B, T, H, cut):
    d = _inputs(cuda_device, B, T, H, seed=T + H)
    o, ht = _fwd(d)
    o1, h1 = _fwd(d, 0, cut)
    o2, h2 = _fwd(d, cut, None, h1)
    assert _same((torch.cat([o1, o2], 1), h2), (o, ht))


@pytest.mark.parametrize("B,T,H", [(1, 8192, 32), (2, 1500, 60)])
def test_stage_calls_take_the_records_of_any_k1(cuda_device, B, T, H):
    """K2 has an argument block of its own: another K2 form, no inputs, outputs elsewhere -- and the inputs' memory may be
    in use for something else by then."""
    d = _inputs(cuda_device, B, T, H, seed=11)
    d["v"] = v = d["v"].clone()
    forms = {0: _Call(d)("kda_fwd").result()}
    for variant in (1, 3, 4):
        forms[variant] = _Call(d, k2_variant=variant)("kda_fwd").result()
    c = _Call(d)("kda_fwd_k1")
    k1_ht, k1_o, k1_v = c.args.ht, c.args.o, c.args.v
    for variant, ref in forms.items():
        c.o.fill_(float("nan")), c.ht.fill_(float("nan"))
        c.args.k2_variant = variant
        c("kda_fwd_k2")
        assert _same(c.result(), ref), variant
    c.args.k2_variant = 0
    # K2 without the inputs
    c.o.fill_(float("nan")), c.ht.fill_(float("nan"))
    c.args.q = c.args.k = c.args.v = c.args.g = c.args.beta = None
    c("kda_fwd_k2")
    assert _same(c.result(), forms[0])
    # the final state and the outputs over what was the values
    c.args.v = k1_v
    states = torch.as_strided(v.view(torch.float32).view(-1), (B, H, D, D), (H * D * D, D * D, D, 1), 4 * D)
    c.args.ht = states.data_ptr()
    c("kda_fwd_k2")
    assert api.check_device_status(c.ws) == 0 and torch.equal(states, forms[0][1])
    c.args.ht, c.args.o = k1_ht, v.data_ptr()
    v.fill_(float("nan"))
    c("kda_fwd_k2")
    assert api.check_device_status(c.ws) == 0 and torch.equal(v, forms[0][0])
    # a state pass over the same records, the values gone
    c.args.o, c.args.k2_variant = k1_o, 1
    c.ht.fill_(float("nan"))
    c("kda_fwd_k2_state", 0)
    assert api.check_device_status(c.ws) == 0 and torch.equal(c.ht, forms[1][1])


def test_k1_for_debugging_and_a_whole_k2(cuda_device):
    """K1 with its debug outputs writes the same records as without."""
    B, T, H = 1, 4097, 16
    d = _inputs(cuda_device, B, T, H, seed=13)
    ref = _Call(d)("kda_fwd").result()
    c = _Call(d, g_out=torch.empty(B, T, H, D, device=cuda_device))
    c("kda_fwd_k1")
    c.args.g_out = None
    assert _same(c("kda_fwd_k2").result(), ref)


@pytest.mark.parametrize("B,T,H,token", [(1, 1087, 96, 50), (1, 8192, 32, 4159), (1, 4096, 16, 63)])
@pytest.mark.parametrize("name", ["q", "k", "v", "g"])
def test_a_token_that_is_not_finite_leaves_earlier_chunks_alone(cuda_device, B, T, H, token, name):
    d = _inputs(cuda_device, B, T, H, seed=17)
    o, ht = _fwd(d)
    d[name][0, token, 1, 7] = float("nan")
    o1, ht1 = _fwd(d)
    first = token // 16 * 16
    others = [h for h in range(H) if h != 1]
    assert o1[0, token, 1].isnan().any()
    assert torch.equal(o1[:, :first, 1], o[:, :first, 1])
    assert torch.equal(o1[:, :, others], o[:, :, others]) and torch.equal(ht1[:, others], ht[:, others])


@pytest.mark.parametrize("H", [75, 96, 148])
def test_forms_that_cannot_wait_for_their_entry_state_are_refused(cuda_device, H):
    """Problems of the tensor-memory form: the flags are there already, so nothing would wait."""
    d = _inputs(cuda_device, 1, 1100, H, seed=19)
    c = _Call(d)("kda_fwd_k1")
    flag = torch.ones(1, dtype=torch.int32, device=cuda_device)
    rc = _lib.load().kda_fwd_k2_after_flags(ctypes.byref(c.args), ctypes.c_void_p(flag.data_ptr()), 1, 1, api._stream_handle())
    torch.cuda.synchronize()
    assert rc == UNSUPPORTED and "wait" in _lib.last_error()
    assert c.o.isnan().all()


# K1 alone in front of K2 and beside it, the general centring (its other instances), packed sequences
@pytest.mark.parametrize("B,T,H,lower_bound,cu", [(1, 33, 2, -5.0, None), (2, 2400, 8, -5.0, None), (1, 100, 3, -8.0, None),
                                                  (1, 50, 2, -5.0, [0, 17, 50])])
def test_gate_parameters_may_be_views_at_any_float(cuda_device, B, T, H, lower_bound, cu):
    d = _inputs(cuda_device, B, T, H, seed=T)
    h0 = None if cu else d["h0"]

    def run(beta, A_log, dt_bias):
        return K.kda_bt16_fwd(d["q"], d["k"], d["v"], d["g"], beta, initial_state=h0, output_final_state=True,
                              use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True,
                              lower_bound=lower_bound, A_log=A_log, dt_bias=dt_bias, cu_seqlens=cu)

    want = run(d["beta"], d["A_log"], d["dt_bias"])
    for shift in (1, 2, 3):
        views = []
        for n in ("beta", "A_log", "dt_bias"):
            flat = torch.full((d[n].numel() + shift,), float("nan"), device=cuda_device)
            flat[shift:] = d[n].flatten()
            views.append(flat[shift:].view(d[n].shape))
        assert _same(run(*views), want)
