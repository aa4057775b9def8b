"""Whole tiles per worker in every order of tiles: row by row and in column-major groups of row tiles."""
import pytest
import torch

from helpers import assert_bit_exact, expected_fp16

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sub(lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nvfp4_gemm_b200 import submission
    return submission


# several waves with a ragged last one and one or two k-tiles (whole tiles win); rows and row groups left over; batches
@pytest.mark.parametrize("raster", [-1, 1, 3, 16])
@pytest.mark.parametrize("shape", [(2300, 2560, 256, 1), (1000, 4608, 512, 2), (700, 5120, 256, 3), (1200, 3968, 256, 2)])
def test_grouped_whole_tiles_cover_the_output_once(sub, oracle, shape, raster):
    from nvfp4_gemm_b200.inputs import generate_input
    data = generate_input(*shape, 91)
    data[6].view(torch.int16).fill_(0x7fff)
    sub.gemm(data, raster=raster)
    sub.check_status()
    assert_bit_exact(data[6], expected_fp16(oracle, data), what=f"{shape} raster {raster} {sub.last_kernel()}")


def test_operands_beyond_l2_take_the_grouped_order_and_the_same_values(sub):
    """117 MB of operands, 1024 tiles of 256 x 256: the groups are the library's own choice."""
    from nvfp4_gemm_b200.inputs import generate_input
    data = generate_input(4096, 4096, 7168, 4, 92)
    data[6].view(torch.int16).fill_(0x7fff)
    sub.custom_kernel(data)
    sub.check_status()
    got = data[6].view(torch.int16).clone()
    data[6].view(torch.int16).fill_(0x7fff)
    sub.gemm(data, raster=-1)
    sub.check_status()
    assert torch.equal(data[6].view(torch.int16), got)
