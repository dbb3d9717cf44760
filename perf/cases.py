"""What the performance of this package is measured on.

The package has two paths: the chunk forward (prefill; ``kda_bt16_fwd``, ``ForwardPlan`` and the
flash-linear-attention adapter ``chunk_kda``) and the token recurrence (decode; ``kda_recurrent_fwd``,
``RecurrentPlan`` and ``fused_recurrent_kda``).  Both are forward only, K = V = 128, bf16 tensors with fp32
beta, gate parameters and states.  A case is one call of one of these entry points.

Keys of a case
  kind      "chunk", "packed" (variable-length sequences in one batch) or "decode"
  api       "fn" (one function call with allocation), "plan" (fixed buffers) or "fla" (the adapter)
  B, T, H   batch, tokens, value heads; Hq q/k heads (grouped value heads when smaller than H)
  g32       the gate arrives as fp32 instead of bf16
  k_first   states are [.., K, V] instead of [.., V, K]
  prepared  gate cumsum, l2-norm and beta sigmoid were done by the caller (the functions' defaults)
  memory    "short": gates as in the benchmark configurations; "long": gates near zero for many heads
  h0        an initial state is given
  nseq, lens_seed   packed only: how many sequences, and what their lengths are drawn from
"""
import math
import random

import torch

import kda_ascendc_b200 as K
from kda_ascendc_b200 import fla_backend

D = 128
BT = 16
LOWER_BOUND = -5.0
MOST_TOKEN_HEADS = 131072 * 16      # of a chunk case: the long-context configuration
MOST_DECODE_HEADS = 256 * 32        # sequences x heads of a decode step


def _case(name, kind, api, B, T, H, Hq=None, g32=False, k_first=False, prepared=False, memory="short", h0=True,
          nseq=0, lens_seed=0):
    c = dict(kind=kind, api=api, B=B, T=T, H=H, Hq=H if Hq is None else Hq, g32=g32, k_first=k_first,
             prepared=prepared, memory=memory, h0=h0, nseq=nseq, lens_seed=lens_seed)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user's decode step: the smallest call there is, all launch and host latency
        _case("decode_b1", "decode", "fn", 1, 1, 32, memory="long"),
        # a small serving batch with everything prepared once, states as flash-linear-attention keeps them
        _case("decode_plan_b8", "decode", "plan", 8, 1, 32, k_first=True, memory="long"),
        # a full serving batch: the states (128 KiB per head, read and written) are the work
        _case("decode_b64", "decode", "fn", 64, 1, 32, memory="long"),
        # checking four drafted tokens per sequence through the adapter
        _case("verify_b16_t4", "decode", "fla", 16, 4, 32, k_first=True, memory="long"),
        # a short prompt, or the odd last piece of a chunked prefill
        _case("prefill_t100", "chunk", "fn", 1, 100, 32, memory="long"),
        # the small benchmark configuration (B2 T1024 H4), gate in fp32 as the reference's function wants it
        _case("prefill_b2_t1024_h4", "chunk", "fn", 2, 1024, 4, g32=True),
        # the middle benchmark configuration on fixed buffers
        _case("plan_b2_t4096_h8", "chunk", "plan", 2, 4096, 8),
        # the headline configuration, and the large-head layer
        _case("prefill_t8192_h32", "chunk", "fn", 1, 8192, 32),
        _case("prefill_t8192_h96", "chunk", "fn", 1, 8192, 96),
        # prompts of very different lengths packed into one call through the adapter
        _case("packed_24_seqs", "packed", "fla", 1, 16411, 32, k_first=True, memory="long", nseq=24, lens_seed=7),
        # a batch of odd length, grouped value heads, the gate and the norms done by the caller's own code
        _case("batch_b8_t2037_gva", "chunk", "fn", 8, 2037, 32, Hq=8, g32=True, prepared=True),
        # the long-context configuration on one GPU: the largest
        _case("long_t131072_h16", "chunk", "plan", 1, 131072, 16, memory="long"),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(("chunk", "decode", "packed"), (5, 3, 2))[0]
    k_first, memory = rng.random() < 0.4, rng.choice(("short", "long"))
    if kind == "decode":
        H = rng.choice((4, 8, 12, 16, 32, 64, 96))
        T = 1 if rng.random() < 0.7 else rng.randint(2, 4)
        B = _log_uniform(rng, 1, min(256, MOST_DECODE_HEADS // (H * T)))
        return _case(None, kind, rng.choice(("fn", "fn", "plan", "fla")), B, T, H, Hq=H // rng.choice((1, 1, 2, 4)),
                     g32=rng.random() < 0.3, k_first=k_first, memory=memory)
    if kind == "packed":
        H = rng.choice((4, 8, 16, 32))
        nseq = _log_uniform(rng, 2, 64)
        T = _log_uniform(rng, 8 * nseq, 32768)
        return _case(None, kind, rng.choice(("fn", "fla")), 1, T, H, g32=rng.random() < 0.3, k_first=k_first,
                     memory=memory, h0=rng.random() < 0.5, nseq=nseq, lens_seed=rng.randrange(1 << 20))
    H = rng.choice((1, 2, 4, 6, 8, 12, 16, 24, 32, 48, 64, 96))
    B = rng.choice((1, 1, 1, 2, 3, 4, 8, 16))
    group = rng.choice((1, 1, 1, 2, 4))
    prepared = rng.random() < 0.15
    g32 = prepared or rng.random() < 0.3
    # no more bytes than the largest listed case: an fp32 gate is a fifth more per token, and there are the states
    most = int(MOST_TOKEN_HEADS * (0.74 if g32 else 0.9))
    T = _log_uniform(rng, 5, min(131072, most // (B * H)))
    return _case(None, kind, "fn" if prepared else rng.choice(("fn", "fn", "plan", "fla")), B, T, H,
                 Hq=H // group if H % group == 0 else H, g32=g32, k_first=k_first, prepared=prepared, memory=memory,
                 h0=rng.random() < 0.7)


def _lengths(case):
    """Lengths of the packed sequences: log-normal shares of the tokens, at least one each."""
    rng = random.Random(case["lens_seed"])
    w = [rng.lognormvariate(0.0, 1.0) for _ in range(case["nseq"])]
    spare = case["T"] - case["nseq"]
    lens = [1 + int(spare * x / sum(w)) for x in w]
    lens[-1] += case["T"] - sum(lens)
    return lens


def _states(case):
    return case["nseq"] if case["kind"] == "packed" else case["B"]


def _chunks(case):
    lens = _lengths(case) if case["kind"] == "packed" else [case["T"]] * case["B"]
    return sum((n + BT - 1) // BT for n in lens)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def rn(*shape):
        return torch.randn(*shape, device="cuda", generator=gen)

    B, T, H, Hq = case["B"], case["T"], case["H"], case["Hq"]
    q, k, v = (rn(B, T, n, D).bfloat16() for n in (Hq, Hq, H))
    g = rn(B, T, H, D)
    if case["memory"] == "long":
        g = g * 0.5 - 1.0
    beta = rn(B, T, H)
    a_log = torch.log(1.0 + 15.0 * torch.rand(H, device="cuda", generator=gen))
    dt_bias = torch.rand(H * D, device="cuda", generator=gen) * 0.2 - 0.1
    h0 = None
    if case["h0"] or case["kind"] == "decode":
        h0 = rn(_states(case), H, D, D) * 0.02
    s = dict(case=case, h0=h0)
    if case["prepared"]:
        # what a caller that does these steps itself hands over: normalised q and k, activated beta and the
        # log2 gate summed within every chunk of 16 tokens
        q, k = (torch.nn.functional.normalize(x.float(), dim=-1).bfloat16() for x in (q, k))
        g = LOWER_BOUND * torch.sigmoid(a_log.exp()[:, None] * (g + dt_bias.view(H, D))) * math.log2(math.e)
        pad = -T % BT
        g = torch.nn.functional.pad(g, (0, 0, 0, 0, 0, pad)).view(B, (T + pad) // BT, BT, H, D).cumsum(2)
        g = g.view(B, T + pad, H, D)[:, :T].contiguous()
        beta = beta.sigmoid()
    elif not case["g32"]:
        g = g.bfloat16()
    s.update(q=q, k=k, v=v, g=g, beta=beta, a_log=a_log, dt_bias=dt_bias)
    if case["kind"] == "packed":
        cu = [0]
        for n in _lengths(case):
            cu.append(cu[-1] + n)
        # a scheduler knows the lengths on the host; the adapter's convention is a tensor for each side
        s["cu"] = torch.tensor(cu, dtype=torch.int32)
        s["cu_gpu"] = s["cu"].cuda()
    if case["api"] == "plan":
        if case["kind"] == "decode":
            s["plan"] = K.RecurrentPlan(q, k, v, g, beta, h0, lower_bound=LOWER_BOUND, A_log=a_log, dt_bias=dt_bias,
                                        state_v_first=not case["k_first"])
        else:
            s["plan"] = K.ForwardPlan(q, k, v, g, beta, initial_state=h0, lower_bound=LOWER_BOUND, A_log=a_log,
                                      dt_bias=dt_bias)
    return s


def run(s):
    c = s["case"]
    if c["api"] == "plan":
        if c["kind"] == "decode":
            return s["plan"].step(), s["plan"].state
        return s["plan"].run()
    args = (s["q"], s["k"], s["v"], s["g"], s["beta"])
    if c["kind"] == "decode":
        if c["api"] == "fla":      # the adapter's convention: the new state comes back as a tensor of its own
            return fla_backend.fused_recurrent_kda(
                *args, A_log=s["a_log"], dt_bias=s["dt_bias"], initial_state=s["h0"], output_final_state=True,
                use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True,
                lower_bound=LOWER_BOUND, transpose_state_layout=not c["k_first"])
        return K.kda_recurrent_fwd(*args, initial_state=s["h0"], inplace_state=True, lower_bound=LOWER_BOUND,
                                   A_log=s["a_log"], dt_bias=s["dt_bias"], state_v_first=not c["k_first"])
    if c["api"] == "fla":
        return fla_backend.chunk_kda(
            *args, initial_state=s["h0"], output_final_state=True, use_qk_l2norm_in_kernel=True,
            use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True, cu_seqlens=s.get("cu_gpu"),
            cu_seqlens_cpu=s.get("cu"), safe_gate=True, lower_bound=LOWER_BOUND, A_log=s["a_log"],
            dt_bias=s["dt_bias"], transpose_state_layout=not c["k_first"])
    if c["prepared"]:
        return K.kda_bt16_fwd(*args, initial_state=s["h0"], output_final_state=True, state_v_first=not c["k_first"])
    return K.kda_bt16_fwd(*args, initial_state=s["h0"], output_final_state=True, use_qk_l2norm_in_kernel=True,
                          use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True, lower_bound=LOWER_BOUND,
                          A_log=s["a_log"], dt_bias=s["dt_bias"], state_v_first=not c["k_first"],
                          cu_seqlens=s.get("cu"))


def work(case):
    tokens = case["B"] * case["T"]
    per_token = case["Hq"] * 2 * D * 2 + case["H"] * (D * 2 + D * (4 if case["g32"] else 2) + 4 + D * 2)
    states = (2 if case["h0"] or case["kind"] == "decode" else 1) * _states(case) * case["H"] * D * D * 4
    if case["kind"] == "decode":
        flops = tokens * case["H"] * 7 * D * D
    else:     # per chunk of 16 tokens and head: two Grams, w and u; two products with the state, its update, A v
        flops = _chunks(case) * case["H"] * (4 * 2 * BT * BT * D + 3 * 2 * BT * D * D + 2 * BT * BT * D)
    return dict(bytes=tokens * per_token + states, flops=flops)


def tolerance(case):
    # o is bf16, and q, k, w and the state are rounded to bf16 on their way into the tensor cores
    return dict(rel=1e-2)
