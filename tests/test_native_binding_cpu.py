"""The native module's translation of the operator's 7-tuple: what it accepts and what it refuses."""
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
