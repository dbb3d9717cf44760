"""Calls one after the other without a wait on the host: each starts ahead of the end of the one before and must not read
what that one still writes."""
import threading

import pytest
import torch

import kda_ascendc_b200 as K
from kda_ascendc_b200 import _lib, api
from oracle import kda_oracle as O
from tests.conftest import to_device

pytestmark = pytest.mark.gpu
FLAGS = dict(use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True, output_final_state=True)


def _inputs(B, T, H, dev):
    d = to_device(O.make_inputs(B, T, H, seed0=T + H, h0_std=0.3), dev)
    d["g"] = (d["g"].float() - 4.0).bfloat16()     # decays that leave much of the state
    return d


def _piece(d, a, b):
    return [d[n][:, a:b].contiguous() for n in ("q", "k", "v", "g", "beta")]


# 8-row, 16-row and tensor-memory K2, one to six chunks a call: every call's initial state is the final state of the one before
@pytest.mark.parametrize("B,H,piece", [(1, 32, 16), (1, 2, 96), (2, 30, 32), (5, 32, 64)])
def test_pieces_of_a_sequence(cuda_device, B, H, piece):
    n = 24
    d = _inputs(B, n * piece, H, cuda_device)
    kw = dict(scale=d["scale"], lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"], **FLAGS)
    pieces = [_piece(d, i * piece, (i + 1) * piece) for i in range(n)]

    def walk(wait):
        h, os = d["initial_state"], []
        for x in pieces:
            o, h = K.kda_bt16_fwd(*x, initial_state=h, **kw)
            if wait:
                torch.cuda.synchronize()
            os.append(o)
        return torch.cat(os, 1), h

    want = walk(True)
    for _ in range(5):
        got = walk(False)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("B,T,k_first", [(1, 1, False), (64, 1, False), (64, 1, True), (16, 4, False), (16, 4, True)])
def test_decode_steps_behind_a_forward(cuda_device, B, T, k_first):
    """A forward, then steps on its final state in place; inputs made on the stream right before each call."""
    H, n = 16, 12
    d = _inputs(B, 32 + n * T, H, cuda_device)
    kw = dict(scale=d["scale"], lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"], state_v_first=not k_first)
    h0 = d["initial_state"].transpose(-1, -2).contiguous() if k_first else d["initial_state"]

    def walk(wait):
        sync = torch.cuda.synchronize if wait else (lambda: None)
        _, h = K.kda_bt16_fwd(*_piece(d, 0, 32), initial_state=h0, **kw, **FLAGS)
        sync()
        os = []
        for i in range(n):
            x = _piece(d, 32 + i * T, 32 + (i + 1) * T)
            sync()
            os.append(K.kda_recurrent_fwd(*x, initial_state=h, inplace_state=True, **kw)[0])
            sync()
        return torch.cat(os, 1), h

    want = walk(True)
    for _ in range(5):
        got = walk(False)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("B,T,H", [(2, 2400, 8), (1, 1991, 19), (1, 1700, 40), (1, 600, 96), (1, 4085, 88)])
def test_two_streams_at_once(cuda_device, B, T, H):
    """Forwards whose K2 runs beside K1 on two streams: each finds the other's CTAs on the SMs that it counted on."""
    runs = []
    for seed in range(2):
        d = _inputs(B, T + 16 * seed, H, cuda_device)
        plan = K.ForwardPlan(d["q"], d["k"], d["v"], d["g"], d["beta"], scale=d["scale"], initial_state=d["initial_state"],
                             lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"])
        plan.run()
        if torch.cuda.get_device_properties(0).multi_processor_count == 148:   # clear, K1 and K2: beside
            assert _lib.load().kda_last_launch_count() == 3
        torch.cuda.synchronize()
        runs.append((plan, torch.cuda.Stream(), plan.o.clone(), plan.final_state.clone()))
    for _ in range(8):
        for plan, stream, _, _ in runs:
            plan.run(stream.cuda_stream)
    torch.cuda.synchronize()
    for plan, _, o, ht in runs:
        assert torch.equal(plan.o, o) and torch.equal(plan.final_state, ht)


def test_reused_workspaces_are_not_shared_by_streams(cuda_device):
    """reuse_workspace=True with one shape on two streams, from two threads: K2 beside K1 and after it."""
    for B, T, H in ((2, 2400, 8), (1, 100, 32), (1, 1616, 32)):
        d = [_inputs(B, T, H, cuda_device) for _ in range(2)]
        d[1]["v"] = d[1]["v"] * -0.5

        def fwd(x):
            return K.kda_bt16_fwd(x["q"], x["k"], x["v"], x["g"], x["beta"], scale=x["scale"], initial_state=x["initial_state"],
                                  lower_bound=x["lower_bound"], A_log=x["A_log"], dt_bias=x["dt_bias"], reuse_workspace=True, **FLAGS)

        want = [fwd(x) for x in d]
        assert not api._WORKSPACE_CACHE
        torch.cuda.synchronize()
        got, streams = [[], []], [torch.cuda.Stream() for _ in d]

        def walk(i):
            with torch.cuda.stream(streams[i]):
                for _ in range(8):
                    got[i].append(fwd(d[i]))

        threads = [threading.Thread(target=walk, args=(i,)) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        for i in range(2):
            assert len(got[i]) == 8
            for o, ht in got[i]:
                assert torch.equal(o, want[i][0]) and torch.equal(ht, want[i][1])


# some sequences long enough for the 16-row launch in front of the tensor-memory one, few of each, and none
@pytest.mark.parametrize("H,chunks", [(16, [300] + [40] * 9), (8, [20] * 12 + [400, 380, 360, 340, 320, 17]), (16, [60] * 11)])
def test_packed_calls_back_to_back_and_on_two_streams(cuda_device, H, chunks):
    cu, n = [0], len(chunks)
    for i, c in enumerate(chunks):
        cu.append(cu[-1] + 16 * c - (i * 5) % 16)
    d = _inputs(1, cu[-1], H, cuda_device)
    gen = torch.Generator(cuda_device).manual_seed(3)
    h0 = torch.randn(n, H, 128, 128, device=cuda_device, generator=gen) * 0.3
    kw = dict(scale=d["scale"], lower_bound=d["lower_bound"], A_log=d["A_log"], dt_bias=d["dt_bias"], **FLAGS)

    def fwd(v, h):
        return K.kda_bt16_fwd(d["q"], d["k"], v, d["g"], d["beta"], initial_state=h, cu_seqlens=cu, **kw)

    fwd(d["v"], h0)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:   # K1, 16-row, tensor-memory
        assert _lib.load().kda_last_launch_count() == 3

    def walk(sign, wait):   # every call's initial states are the final states of the one before, its values made right before it
        h, os = h0, []
        for i in range(4):
            o, h = fwd(d["v"] * (sign * (i + 1)), h)
            if wait:
                torch.cuda.synchronize()
            os.append(o)
        return os, h

    want = [walk(sign, True) for sign in (1.0, -0.5)]
    streams = [torch.cuda.Stream() for _ in want]
    torch.cuda.synchronize()
    got = [walk(1.0, False)]
    for stream, sign in zip(streams, (1.0, -0.5)):
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            got.append(walk(sign, False))
    torch.cuda.synchronize()
    for g, w in zip(got, (want[0], *want)):
        assert all(torch.equal(a, b) for a, b in zip(g[0], w[0])) and torch.equal(g[1], w[1])


# K1 after K2's set-up only, beside K2 in either register form and in tensor memory
@pytest.mark.parametrize("B,T,H", [(1, 100, 32), (2, 2400, 8), (1, 1630, 32), (1, 600, 96)])
@pytest.mark.parametrize("front", ["memset", "copy", "event", "join"])
def test_captured_forward_and_decode_steps_behind_any_node(cuda_device, B, T, H, front):
    """A graph in which the node in front of the forward is a memset, a copy, an event of another stream or a join of two
    streams, and token steps on the forward's final state come behind it; replayed on changing values."""
    d = _inputs(B, T + 2, H, cuda_device)
    x = [t.clone() for t in _piece(d, 0, T)]
    src = x[2].clone()
    toks = [_piece(d, T + i, T + i + 1) for i in range(2)]
    plan = K.ForwardPlan(*x, scale=d["scale"], initial_state=d["initial_state"], lower_bound=d["lower_bound"], A_log=d["A_log"],
                         dt_bias=d["dt_bias"])
    steps = [K.RecurrentPlan(*t, plan.final_state, scale=d["scale"], lower_bound=d["lower_bound"], A_log=d["A_log"],
                             dt_bias=d["dt_bias"]) for t in toks]
    v, outs = x[2], [torch.empty_like(steps[0].o) for _ in steps]

    def body(main, other):
        if front in ("memset", "copy"):
            v.zero_() if front == "memset" else v.copy_(src)
        else:
            if other is not None:
                other.wait_stream(main)
            with torch.cuda.stream(main if other is None else other):
                v.copy_(src)
                v.mul_(-0.5)
            y = src * 2 if front == "join" else None   # a kernel on this stream too
            if other is not None:
                main.wait_stream(other)
            if y is not None:
                v.add_(y)
        plan.run()
        for s, o in zip(steps, outs):
            s.step()
            o.copy_(s.o)

    body(torch.cuda.current_stream(), None)
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        body(torch.cuda.current_stream(), torch.cuda.Stream())
    for i in range(3):
        src.mul_(-0.75)
        torch.cuda.synchronize()
        v.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in (plan.o, plan.final_state, *outs)]
        body(torch.cuda.current_stream(), None)
        assert all(t.isfinite().all() for t in got)
        assert all(torch.equal(a, b) for a, b in zip(got, (plan.o, plan.final_state, *outs)))
    del graph
