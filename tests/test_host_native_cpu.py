"""The native host path (csrc/kda_host.cpp) without a GPU: what it does with errors and with calls it leaves to the
Python path.  The inputs are wrapper tensors that report a CUDA device and have no memory; every call here ends before
anything is allocated or launched."""
import subprocess
import sys
import textwrap
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

PRELUDE = """
import torch
from kda_ascendc_b200 import _lib

class OnCuda(torch.Tensor):   # says it lives on a GPU; every operation on it raises `error`
    error = RuntimeError("an operation ran")
    @staticmethod
    def __new__(cls, *size, dtype=torch.float32, **kw):
        return torch.Tensor._make_wrapper_subclass(cls, size, dtype=dtype, **dict(dict(device="cuda:0"), **kw))
    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        raise cls.error

bf, H = torch.bfloat16, 2
def chunk_args(**kw):
    a = dict(q=OnCuda(1, 32, H, 128, dtype=bf), k=OnCuda(1, 32, H, 128, dtype=bf), v=OnCuda(1, 32, H, 128, dtype=bf),
             g=OnCuda(1, 32, H, 128), beta=OnCuda(1, 32, H), scale=None, initial_state=None, output_final_state=True,
             l2norm=True, gate=True, beta_sigmoid=True, safe_gate=True, lower_bound=-5.0, A_log=OnCuda(H), dt_bias=None,
             state_v_first=True, cu_seqlens=None, fla=False)
    assert set(kw) <= set(a)
    return list(dict(a, **kw).values())
"""


def run(body):
    """Run the body in an interpreter of its own (a lost interpreter lock ends the process)."""
    r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(body)], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout[-1000:], r.stderr[-3000:])


def test_an_exception_outside_the_interpreter_lock_reaches_the_caller():
    """Offsets on a GPU are read without the lock; that read can fail (a capturing stream, an earlier CUDA error)."""
    run("""
        for _ in range(2):
            try:
                _lib.host().chunk(*chunk_args(cu_seqlens=OnCuda(3, dtype=torch.int32)))
            except RuntimeError:
                pass
            else:
                raise SystemExit("no exception")
    """)


def test_exceptions_keep_their_type_and_message():
    """What PyTorch raises under the native call arrives as it would from the Python path."""
    run("""
        for OnCuda.error in (RuntimeError("an operation ran"), torch.OutOfMemoryError("no room"), KeyError(7)):
            try:
                _lib.host().chunk(*chunk_args(cu_seqlens=OnCuda(3, dtype=torch.int32)))
            except Exception as e:
                assert type(e) is type(OnCuda.error) and str(e) == str(OnCuda.error), repr(e)
            else:
                raise SystemExit("no exception")
    """)


def test_a_number_that_does_not_fit_is_left_to_the_python_path():
    """No launch with a value that is not the caller's, and no exception left pending."""
    run("""
        for bad in (dict(scale=10**400), dict(lower_bound=-10**400), dict(lower_bound=10**400)):
            assert _lib.host().chunk(*chunk_args(**bad)) is None, bad
    """)


def test_both_paths_refuse_the_same_calls():
    """The argument rules stand twice, in api.py / fla_backend.py and in kda_host.cpp: every call that the Python rules
    refuse is left to them by the native path, and a call that they accept is taken by it."""
    run("""
        import kda_ascendc_b200 as K
        from kda_ascendc_b200 import api, fla_backend
        host = _lib.host()
        def tensor(name, *size, **kw):
            return {name: OnCuda(*size, **kw)}
        both = [                       # tensors, with the shapes of chunk_args (B 1, T 32, H 2)
            *(tensor(n, 32, H, 128, dtype=bf) for n in "qkvg"), tensor("beta", 1, 32),
            *(tensor(n, 1, 32, H, 128) for n in "qkv"), tensor("g", 1, 32, H, 128, dtype=torch.float16),
            tensor("beta", 1, 32, H, dtype=bf), tensor("beta", 1, 32, 3),
            *(tensor(n, 1, 16, H, 128, dtype=bf) for n in "qkvg"), *(tensor(n, 1, 32, 3, 128, dtype=bf) for n in "qkvg"),
            *(tensor(n, 1, 32, H, 64, dtype=bf) for n in "qkvg"), *(tensor(n, 1, 0, H, 128, dtype=bf) for n in "qkvg"),
            *(tensor(n, 1, 32, H, 128, dtype=bf, device="cuda:1") for n in "kvg"), tensor("beta", 1, 32, H, device="cuda:1"),
            *(tensor(n, 1, 32, H, 128, dtype=bf, strides=(32 * H * 128, H * 128, 1, H)) for n in "qkvg"),
            tensor("initial_state", 2, H, 128, 128), tensor("initial_state", 1, H, 128, 64),
            tensor("initial_state", 1, H, 128, 128, dtype=bf), tensor("initial_state", 1, H, 128, 128, device="cuda:1"),
            tensor("initial_state", 1, H, 128, 128, strides=(H << 14, 1 << 14, 1, 128)),
            tensor("A_log", 3), tensor("A_log", H, dtype=bf), tensor("A_log", H, device="cuda:1"), dict(A_log=None),
            tensor("A_log", H, strides=(2,)), tensor("dt_bias", H * 128 + 1), tensor("dt_bias", H * 128, dtype=bf),
            tensor("dt_bias", H * 128, device="cuda:1"), tensor("dt_bias", H * 128, strides=(2,)),
            *(dict(lower_bound=x) for x in (-11.0, 0.0, 1, float("nan")))]
        chunk_only = [dict(safe_gate=False), dict(lower_bound=None),
                      *(tensor(n, 1, 32, H, 128, dtype=bf, strides=(64 * H * 128, 2 * H * 128, 128, 1)) for n in "qkvg"),
                      tensor("beta", 1, 32, H, strides=(64 * H, 2 * H, 1))]
        names = "q k v g beta scale initial_state output_final_state l2norm gate beta_sigmoid safe_gate lower_bound A_log " \
                "dt_bias state_v_first cu_seqlens fla".split()
        def refused(f, *args, **kw):
            try:
                f(*args, **kw)
            except (ValueError, TypeError, NotImplementedError):
                return True
            raise SystemExit("not refused")
        def accepted(f, *args):   # taken: it ends at the device that is not there, or at the pointers, which are null
            try:
                r = f(*args)
            except (RuntimeError, ValueError) as e:
                return "CUDA" in str(e) or "required" in str(e) or "needs q" in str(e)
            raise SystemExit(f"returned {r}")
        for bad in both + chunk_only:
            a = dict(zip(names, chunk_args(**bad)))
            assert host.chunk(*a.values()) is None, bad
            kw = {k: a[k] for k in "initial_state output_final_state safe_gate lower_bound A_log dt_bias".split()}
            five = [a[k] for k in ("q", "k", "v", "g", "beta")]
            assert refused(K.kda_bt16_fwd, *five, use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True,
                           use_beta_sigmoid_in_kernel=True, **kw), bad
        five = lambda a: [a[k] for k in ("q", "k", "v", "g", "beta")]
        def recurrent_args(a, inplace=False, fla=False):
            return (*five(a), None, a["initial_state"], True, a["lower_bound"], a["A_log"], a["dt_bias"], inplace, True, 4, fla)
        for bad in both:
            a = dict(zip(names, chunk_args(**bad)))
            assert host.recurrent(*recurrent_args(a)) is None, bad
            assert refused(K.kda_recurrent_fwd, *five(a), initial_state=a["initial_state"], lower_bound=a["lower_bound"],
                           A_log=a["A_log"], dt_bias=a["dt_bias"]), bad
        a = dict(zip(names, chunk_args()))
        assert host.recurrent(*recurrent_args(a, inplace=True)) is None
        assert refused(K.kda_recurrent_fwd, *five(a), A_log=a["A_log"], inplace_state=True)
        # the adapter: no autograd through the call
        for n in ("q", "k", "v"):
            a = dict(zip(names, chunk_args(**tensor(n, 1, 32, H, 128, dtype=bf, requires_grad=True), fla=True)))
            assert host.chunk(*a.values()) is None and host.recurrent(*recurrent_args(a, fla=True)) is None
            kw = dict(use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, lower_bound=-5.0, A_log=a["A_log"])
            assert refused(fla_backend.chunk_kda, *five(a), safe_gate=True, **kw)
            assert refused(fla_backend.fused_recurrent_kda, *five(a), use_beta_sigmoid_in_kernel=True, **kw)
            with torch.no_grad():
                assert accepted(host.chunk, *a.values()) and accepted(host.recurrent, *recurrent_args(a, fla=True))
        # packed sequences
        for cu in ([0, 16], [0], [], [0, 33], [0, 20, 10, 32], [0, 16, 16, 32], [1, 32], [-1, 32], torch.tensor([[0, 32]])):
            assert host.chunk(*chunk_args(cu_seqlens=cu)) is None, cu
            assert refused(api._varlen_tables, cu, 32, H, "cpu"), cu
        # accepted
        for good in ({}, dict(scale=1), dict(scale=0.5, cu_seqlens=[0, 1, 32]), dict(cu_seqlens=torch.tensor([0, 32])),
                     dict(gate=False, A_log=None, lower_bound=None), tensor("initial_state", 1, H, 128, 128),
                     tensor("dt_bias", H * 128), dict(tensor("dt_bias", H, 128), fla=True),
                     dict(q=OnCuda(1, 32, 1, 128, dtype=bf), k=OnCuda(1, 32, 1, 128, dtype=bf))):
            assert accepted(host.chunk, *chunk_args(**good)), good
        for good in ({}, tensor("beta", 1, 32, H, strides=(64 * H, 2 * H, 1)), tensor("initial_state", 1, H, 128, 128),
                     *(tensor(n, 1, 32, H, 128, dtype=bf, strides=(64 * H * 128, 2 * H * 128, 128, 1)) for n in "qkvg")):
            assert accepted(host.recurrent, *recurrent_args(dict(zip(names, chunk_args(**good))))), good
    """)
