"""The tensor-memory (tcgen05) organisation of K2 against the oracle and against the mma.sync
organisations.  Same tolerances as the default path: o 1e-3, state 2e-3 on benchmark-distributed
inputs; the reference's relative 2e-2 bound where states are O(1)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import kda_oracle as O  # noqa: E402


def _run(inp, variant, cu=None):
    from kda_ascendc_b200 import api
    dev = torch.device("cuda", 0)
    d = {k: (v.to(dev) if torch.is_tensor(v) else v) for k, v in inp.items()}
    o, ht = api._forward(d["q"], d["k"], d["v"], d["g"], d["beta"], d["scale"], d["initial_state"], True, True, True, True,
                         d["lower_bound"], d["A_log"], d["dt_bias"], True, k2_variant=variant, cu_seqlens=cu)
    torch.cuda.synchronize()
    return o.float().cpu(), ht.cpu()


@pytest.mark.parametrize("B,T,H,h0_std", [(1, 16, 1, None), (2, 1000, 4, 0.02), (1, 333, 3, 0.0), (5, 64, 40, 0.02)])
def test_tensor_memory_k2_matches_oracle(B, T, H, h0_std):
    inp = O.make_inputs(B, T, H, seed0=17, h0_std=h0_std)
    o, ht = _run(inp, 4)
    o_r, ht_r = O.run_chunk_reference(inp)
    assert (o - o_r.float()).abs().max().item() <= 1e-3
    assert (ht - ht_r).abs().max().item() <= 2e-3
    o1, ht1 = _run(inp, 1)
    assert (o - o1).abs().max().item() <= 2.5e-4       # one bf16 step of |o| <= 0.06
    assert (ht - ht1).abs().max().item() <= 2e-5


@pytest.mark.parametrize("regime,h0_std", [("carry", 0.5), ("long_memory", 0.3)])
def test_tensor_memory_k2_carries_the_state(regime, h0_std):
    inp = O.make_inputs(2, 512, 3, seed0=23, regime=regime, h0_std=h0_std)
    o, ht = _run(inp, 4)
    o_r, ht_r = O.run_chunk_reference(inp)
    assert (o - o_r.float()).abs().max().item() <= 2e-2 * o_r.float().abs().max().item()
    assert (ht - ht_r).abs().max().item() <= 2e-2 * ht_r.abs().max().item()
    o1, ht1 = _run(inp, 3)
    assert (ht - ht1).abs().max().item() <= 1e-3 * ht_r.abs().max().item()


def test_tensor_memory_k2_packed_sequences():
    lengths = [40, 1, 17, 160, 31]
    T = sum(lengths)
    inp = O.make_inputs(1, T, 3, seed0=29, h0_std=None)
    g = torch.Generator().manual_seed(5)
    inp["initial_state"] = torch.randn(len(lengths), 3, 128, 128, generator=g) * 0.05
    cu = [0]
    for L in lengths:
        cu.append(cu[-1] + L)
    o, ht = _run(inp, 4, cu=cu)
    o_r, ht_r = O.run_chunk_reference_varlen(inp, cu)
    assert (o - o_r.float()).abs().max().item() <= 1e-3
    assert (ht - ht_r).abs().max().item() <= 2e-3


def test_tail_wave_runs_in_an_mma_sync_form():
    """320 chains on 148 SMs: 296 fill one wave of the tensor-memory form, the other 24 follow in
    the 8-row mma.sync form (a second K2 launch on the chains' sub-range).  Both halves against the oracle."""
    from kda_ascendc_b200 import _lib
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B, T, H = 10, 72, 32
    inp = O.make_inputs(B, T, H, seed0=31, h0_std=0.02)
    o, ht = _run(inp, 0)
    launches = _lib.load().kda_last_launch_count()
    tail = (B * H) % (2 * sms)
    if B * H > 2 * sms and 0 < tail * 2 <= sms:
        assert launches == 3     # K1, K2 on tcgen05 for the full waves, K2 on mma.sync for the tail
    o_r, ht_r = O.run_chunk_reference(inp)
    assert (o - o_r.float()).abs().max().item() <= 1e-3
    assert (ht - ht_r).abs().max().item() <= 2e-3
    o3, ht3 = _run(inp, 3)
    assert (o - o3).abs().max().item() <= 2.5e-4
    assert (ht - ht3).abs().max().item() <= 2e-5
    # the tail chains are the last ones: bit-identical to the form that ran them (8-row up to SMs/4 chains)
    first_tail = B * H - tail
    if B * H > 2 * sms and 0 < tail * 2 <= sms:
        ref = _run(inp, 1)[1] if tail * 4 <= sms else ht3
        assert torch.equal(ht.reshape(B * H, 128, 128)[first_tail:], ref.reshape(B * H, 128, 128)[first_tail:])


def test_tail_wave_with_packed_sequences():
    """20 packed sequences x 16 heads = 320 chains: the automatic choice (tensor memory + tail in the
    16-row form) against the 16-row form alone."""
    lengths = [64 + 7 * i for i in range(20)]
    T, H = sum(lengths), 16
    inp = O.make_inputs(1, T, H, seed0=37, h0_std=None)
    g = torch.Generator().manual_seed(7)
    inp["initial_state"] = torch.randn(len(lengths), H, 128, 128, generator=g) * 0.05
    cu = [0]
    for L in lengths:
        cu.append(cu[-1] + L)
    o, ht = _run(inp, 0, cu=cu)
    o3, ht3 = _run(inp, 3, cu=cu)
    assert (o - o3).abs().max().item() <= 2.5e-4
    assert (ht - ht3).abs().max().item() <= 2e-5
    o_r, ht_r = O.run_chunk_reference_varlen(inp, cu)
    assert (o - o_r.float()).abs().max().item() <= 1e-3
    assert (ht - ht_r).abs().max().item() <= 2e-3


# chains are taken longest sequence first, up to 256 sequences: ties, one-token sequences, and the line itself
@pytest.mark.parametrize("lengths,H", [([65] * 10, 16), ([1, 300, 17, 300, 16, 64, 1, 299, 33, 128], 16), ([5, 700] * 11, 15),
                                       ([70 + i % 9 for i in range(256)], 1), ([70 + i % 9 for i in range(257)], 1)])
def test_longest_sequence_first(lengths, H):
    T = sum(lengths)
    inp = O.make_inputs(1, T, H, seed0=41, h0_std=None)
    g = torch.Generator().manual_seed(8)
    inp["initial_state"] = torch.randn(len(lengths), H, 128, 128, generator=g) * 0.05
    cu = [0]
    for L in lengths:
        cu.append(cu[-1] + L)
    o, ht = _run(inp, 0, cu=cu)
    o4, ht4 = _run(inp, 4, cu=cu)
    o3, ht3 = _run(inp, 3, cu=cu)
    for a, b in ((o, o3), (o4, o3)):
        assert (a - b).abs().max().item() <= 2.5e-4
    for a, b in ((ht, ht3), (ht4, ht3)):
        assert (a - b).abs().max().item() <= 2e-5


# the chain at a place is picked bit by bit: lengths of one to seven bits with many ties, eight lengths per lane; and
# both sides of the line in chains (4 x SMs x mean chunks), above which the chains keep their own order
@pytest.mark.parametrize("n,lo,hi,H", [(2, 1, 600, 150), (33, 1, 1500, 9), (255, 1, 64, 2), (256, 20, 40, 4), (256, 20, 40, 5)])
def test_any_lengths_longest_first(n, lo, hi, H):
    g = torch.Generator().manual_seed(n + H)
    lengths = torch.randint(lo, hi + 1, (n,), generator=g).tolist()
    inp = O.make_inputs(1, sum(lengths), H, seed0=43, h0_std=None)
    inp["initial_state"] = torch.randn(n, H, 128, 128, generator=g) * 0.05
    cu = [0]
    for L in lengths:
        cu.append(cu[-1] + L)
    o, ht = _run(inp, 4, cu=cu)
    o3, ht3 = _run(inp, 3, cu=cu)
    assert (o - o3).abs().max().item() <= 2.5e-4       # one bf16 step of |o| <= 0.06, as above
    assert (ht - ht3).abs().max().item() <= 2e-5


def test_any_number_of_chunks_around_the_stages():
    """One chunk to more than twice the four stages: every length gives the bits of the longest one's first chunks."""
    inp = O.make_inputs(2, 16 * 9 - 3, 3, seed0=29, regime="carry", h0_std=0.3)
    want, _ = _run(inp, 4)
    for n in range(1, 9):
        part = {k: v[:, :16 * n].contiguous() if k in ("q", "k", "v", "g", "beta") else v for k, v in inp.items()}
        for _ in range(2):
            o, ht = _run(part, 4)
            assert torch.equal(o, want[:, :16 * n])
        rest = {k: v[:, 16 * n:].contiguous() if k in ("q", "k", "v", "g", "beta") else v for k, v in inp.items()}
        o, _ = _run(dict(rest, initial_state=ht.cpu()), 4)
        assert torch.equal(o, want[:, 16 * n:])
