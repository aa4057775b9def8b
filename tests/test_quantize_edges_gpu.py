"""The quantiser where its launch shape or its accesses change, and on values that are no numbers."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _quantize(lib, x, row_stride):
    from nvfp4_gemm_b200 import _lib
    rows, k = x.shape
    packed = torch.full((rows, k // 2), 0xEE, dtype=torch.uint8, device="cuda")
    sf = torch.full((rows, k // 16), 0xEE, dtype=torch.uint8, device="cuda")
    perm = torch.full(((rows + 127) // 128, (k // 64) * 512), 0xEE, dtype=torch.uint8, device="cuda")
    _lib.check(lib.nvfp4_quantize(x.data_ptr(), int(x.dtype == torch.bfloat16), packed.data_ptr(), sf.data_ptr(), perm.data_ptr(),
                                  rows, k, row_stride, k // 2, k // 16, torch.cuda.current_stream().cuda_stream))
    return packed, sf, perm


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("offset", [0, 8])          # x 32-byte aligned, and 16-byte aligned only
@pytest.mark.parametrize("rows,k", [(8161, 7232), (8193, 7168), (33, 576), (7, 512)])
def test_large_and_ragged_inputs_equal_small_pieces_and_the_oracle(lib, oracle, dtype, offset, rows, k):
    """The first two sizes take four rows per warp, with rows and columns left over; quantised 128 rows at
    a time they take one.  Every row is quantised by itself, so the pieces have the same bytes."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    buf = torch.randn(rows * k + offset, generator=g, device="cuda", dtype=dtype)
    x = buf[offset:].view(rows, k)
    packed, sf, perm = _quantize(lib, x, k)
    for r in range(0, rows, 128):
        part = x[r:r + 128]
        p, s, q = _quantize(lib, part, k)
        assert torch.equal(packed[r:r + 128], p) and torch.equal(sf[r:r + 128], s) and torch.equal(perm[r // 128], q[0])
    for part, codes, scales in ((x[:40], packed[:40], sf[:40]), (x[-40:], packed[-40:], sf[-40:])):
        exp_codes, exp_scales = oracle.quantize_rows(part.float().cpu().numpy())
        assert np.array_equal(codes.cpu().numpy(), exp_codes) and np.array_equal(scales.cpu().numpy(), exp_scales)
    last = rows % 128
    if last:                                         # rows that do not exist have zero scales
        atoms = perm[-1].view(k // 64, 32, 4, 4).permute(2, 1, 0, 3).reshape(128, k // 16)
        assert int(atoms[last:].sum()) == 0 and torch.equal(atoms[:last], sf[-last:])


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_values_that_are_no_numbers(lib, dtype):
    """A NaN does not count towards its block's scale; it becomes +6 where the rest is within 65504 and
    -6 where the rest is not.  Infinities saturate the scale and the element."""
    x = torch.zeros((1, 64), dtype=dtype, device="cuda")
    x[0, 0], x[0, 1], x[0, 2] = 6.0, float("nan"), -3.0            # scale 1
    x[0, 16], x[0, 17], x[0, 18] = float("inf"), float("nan"), 2688.0   # scale 448
    x[0, 32], x[0, 33] = -float("inf"), -224.0                     # scale 448: -0.5
    x[0, 48] = float("nan")                                        # nothing else: scale 0, all codes 0
    packed, sf, _ = _quantize(lib, x, 64)
    assert sf[0].tolist() == [0x38, 0x7E, 0x7E, 0x00]
    codes = packed[0].cpu().numpy()
    nibbles = np.stack([codes & 15, codes >> 4], axis=-1).reshape(4, 16)
    assert nibbles[0, :4].tolist() == [0x7, 0x7, 0xD, 0x0]
    assert nibbles[1, :4].tolist() == [0x7, 0xF, 0x7, 0x0]
    assert nibbles[2, :3].tolist() == [0xF, 0x9, 0x0]
    assert not nibbles[3].any()


def test_back_to_back_launches_respect_stream_order(lib):
    """The quantiser may start before the kernel ahead of it has ended: its input is rewritten in place right
    before each launch, and its outputs are read right after."""
    rows, k = 2048, 7168
    g = torch.Generator(device="cuda").manual_seed(5)
    inputs = [torch.randn((rows, k), generator=g, device="cuda", dtype=torch.bfloat16) * 2.0 ** i for i in range(3)]
    exp = []
    for x in inputs:
        exp.append([t.clone() for t in _quantize(lib, x, k)])
        torch.cuda.synchronize()
    work = torch.empty_like(inputs[0])
    outs = []
    for _ in range(5):
        for x in inputs:
            work.copy_(x)
            outs.append([t.clone() for t in _quantize(lib, work, k)])
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        for got, e in zip(o, exp[i % 3]):
            assert torch.equal(got, e), i
