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
    def __new__(cls, *size, dtype=torch.float32):
        return torch.Tensor._make_wrapper_subclass(cls, size, dtype=dtype, device="cuda:0")
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
