"""The native module's translation of the operator's 7-tuple: what it accepts and what it refuses."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from nvfp4_gemm_b200.inputs import generate_input
from nvfp4_gemm_b200.submission import custom_kernel, gemm_epilogue, make_problem


def test_a_list_and_a_strided_view_translate_like_the_tuple(lib):
    data = generate_input(130, 256, 512, 2, 1, device="cpu")
    p, q = make_problem(data), make_problem(list(data))
    assert bytes(p) == bytes(q)
    wide = torch.empty((2, 130, 300), dtype=torch.float16).permute(1, 2, 0)
    r = make_problem(data[:6] + (wide[:, 8:264],))
    assert (r.c_row_stride, r.c_batch_stride, r.c) == (300, 130 * 300, wide.data_ptr() + 16)


@pytest.mark.parametrize("change,error,text", [
    (lambda d: d[:6], ValueError, "seven"),
    (lambda d: (d[0], d[1][:, :64]) + d[2:], ValueError, "disagree"),
    (lambda d: d[:6] + (d[6][:64],), ValueError, "expected"),
    (lambda d: d[:6] + (d[6].float(),), ValueError, "fp16 output"),
    (lambda d: (d[0].view(torch.uint8)[:, ::2],) + d[1:], ValueError, "disagree"),
    (lambda d: (d[0][:, :, 0],) + d[1:], ValueError, "three dimensions"),
    (lambda d: d[:4] + (d[2],) + d[5:], IndexError, "batch dimension"),
    (lambda d: (1,) + d[1:], TypeError, "tensor"),
])
def test_malformed_tuples_are_refused(lib, change, error, text):
    data = generate_input(128, 256, 512, 1, 1, device="cpu")
    with pytest.raises(error, match=text):
        make_problem(change(data))


def test_entry_points_refuse_cpu_tensors(lib):
    data = generate_input(128, 256, 256, 1, 1, device="cpu")
    for call in (custom_kernel, gemm_epilogue, lambda d: custom_kernel(list(d))):
        with pytest.raises(ValueError, match="no CPU fallback"):
            call(data)


_ON_NO_DEVICE = """
from collections import UserList
import torch
from nvfp4_gemm_b200 import submission

class Elsewhere(torch.Tensor):
    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        raise AssertionError(func)

def tensor(rows, cols, dtype):
    return torch.Tensor._make_wrapper_subclass(Elsewhere, (rows, cols, 1), strides=(cols, 1, rows * cols), dtype=dtype, device="cuda:63")

data = (tensor(128, 128, torch.uint8), tensor(256, 128, torch.uint8), None, None, None, None, tensor(128, 256, torch.float16))
for call in (submission.custom_kernel, submission.gemm_epilogue):
    try:
        call(data)
    except RuntimeError as e:
        print("refused:", type(e).__name__)
"""
_OUT_IN_A_SEQUENCE = """
out = UserList([tensor(128, 128, torch.uint8), tensor(128, 16, torch.uint8), tensor(128, 16, torch.uint8)])
try:
    submission.gemm_epilogue(data, nvfp4_out=True, out=out)
except RuntimeError as e:
    print("accepted")
"""


def _run(text):
    return subprocess.run([sys.executable, "-c", text], cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True, timeout=300)


def test_a_cuda_error_ahead_of_the_call_is_a_python_exception(lib):
    """Tensors that say they are on a device which no machine has: making it current fails, inside the
    native module.  (In a process of its own: the failure to guard against is a crash.)"""
    r = _run(_ON_NO_DEVICE)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.splitlines() == ["refused: RuntimeError"] * 2


def test_out_may_be_any_sequence(lib):
    """The three tensors are taken from whatever sequence holds them; the call then fails at the device, not before."""
    r = _run(_ON_NO_DEVICE + _OUT_IN_A_SEQUENCE)
    assert r.returncode == 0 and r.stdout.splitlines()[-1] == "accepted", r.stderr[-2000:]
