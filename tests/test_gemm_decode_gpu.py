"""The decode kernel (few rows): every tile width, split of K and ring depth, at the edges of its tiles."""
import pytest
import torch

from helpers import assert_bit_exact, expected_fp16

pytestmark = pytest.mark.gpu

# (shape, kernel that the launch code picks on 148 SMs)
CASES = [
    ((1, 128, 256, 1), "gemm_decode_t32_s8"), ((32, 4864, 2304, 1), "gemm_decode_t32_s8"), ((17, 384, 1792, 2), "gemm_decode_t32_s8"),
    ((31, 2560, 3072, 1), "gemm_splitk2_decode_t32"), ((7, 128, 2048, 3), "gemm_splitk4_decode_t32"), ((32, 256, 12288, 1), "gemm_splitk8_decode_t32"),
    ((5, 19072, 256, 1), "gemm_decode_t32_s4"), ((32, 6400, 1536, 3), "gemm_decode_t32_s4"),
    ((33, 256, 1024, 1), "gemm_decode_t64_s7"), ((64, 4864, 2304, 1), "gemm_decode_t64_s7"),
    ((63, 2560, 3328, 1), "gemm_splitk2_decode_t64"), ((64, 256, 2304, 2), "gemm_splitk4_decode_t64"), ((50, 128, 12800, 1), "gemm_splitk8_decode_t64"),
    ((40, 6400, 512, 3), "gemm_decode_t64_s3"), ((64, 19072, 1280, 1), "gemm_decode_t64_s3"),
    ((65, 2560, 3072, 1), "gemm_splitk2_decode_t128"), ((128, 2432, 4352, 2), "gemm_splitk2_decode_t128"),
    ((97, 256, 3328, 2), "gemm_splitk4_decode_t128"), ((127, 128, 12288, 1), "gemm_splitk8_decode_t128"), ((128, 256, 12544, 1), "gemm_splitk8_decode_t128"),
    ((129, 1280, 4096, 1), "gemm_splitk2_decode_t128"), ((300, 384, 3072, 2), "gemm_splitk4_decode_t128"), ((256, 128, 12288, 4), "gemm_splitk8_decode_t128"),
]


@pytest.fixture(scope="module")
def sub(lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nvfp4_gemm_b200 import submission
    return submission


@pytest.mark.parametrize("shape,kernel", CASES)
def test_decode_matches_oracle_bit_exact(sub, oracle, shape, kernel):
    """fp32 sums of these inputs are exact in any order, so the fp16 results are equal."""
    from nvfp4_gemm_b200.inputs import generate_input
    data = generate_input(*shape, 77)
    exp = expected_fp16(oracle, data)
    for _ in range(2):
        data[6].view(torch.int16).fill_(0x7fff)        # NaN canary: every element must be written
        sub.custom_kernel(data)
        sub.check_status()
        if torch.cuda.get_device_properties(0).multi_processor_count == 148:
            assert sub.last_kernel() == kernel
        assert_bit_exact(data[6], exp, what=f"{shape} {sub.last_kernel()}")


# many tiles per SM: where the persistent kernels take over
@pytest.mark.parametrize("shape,decode", [((17, 25344, 512, 3), False), ((17, 25344, 1024, 3), True), ((50, 19072, 512, 2), False), ((50, 18944, 512, 2), True)])
def test_many_tiles(sub, oracle, shape, decode):
    from nvfp4_gemm_b200.inputs import generate_input
    data = generate_input(*shape, 79)
    data[6].view(torch.int16).fill_(0x7fff)
    sub.custom_kernel(data)
    sub.check_status()
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert ("decode" in sub.last_kernel()) == decode
    assert_bit_exact(data[6], expected_fp16(oracle, data), what=f"{shape} {sub.last_kernel()}")


@pytest.mark.parametrize("shape,kernel", CASES)
def test_decode_epilogue_equals_the_persistent_kernels(sub, shape, kernel):
    """Bias, ReLU and re-quantising give the bytes that the 128-row-tile kernels give; rows of the last
    scale block that do not exist read as zero scales."""
    from nvfp4_gemm_b200.inputs import generate_input
    m, n, k, l = shape
    data = generate_input(*shape, 78)[:6] + (None,)
    bias = (torch.randn(n, generator=torch.Generator().manual_seed(4)) * 64).half().cuda()
    got = sub.gemm_epilogue(data, bias=bias, activation="relu", nvfp4_out=True)
    for t in got:
        t.view(torch.uint8).fill_(0xA5)
    sub.gemm_epilogue(data, bias=bias, activation="relu", nvfp4_out=True, out=got)
    sub.check_status()
    assert "decode" in sub.last_kernel()
    exp = sub.gemm_epilogue(data, bias=bias, activation="relu", nvfp4_out=True, split_k=1)
    sub.check_status()
    assert "decode" not in sub.last_kernel()
    for g, e in zip(got, exp):
        assert torch.equal(g.view(torch.uint8), e.view(torch.uint8)), f"{shape} {kernel}"
    blocks = (m + 127) // 128
    flat = torch.as_strided(got[2].view(torch.uint8), (l, blocks, n // 64, 32, 4, 4),       # [l][row block][atom][row % 32][row / 32][scale]
                            (blocks * n // 64 * 512, n // 64 * 512, 512, 16, 4, 1))
    rows = flat.permute(0, 1, 4, 3, 2, 5).reshape(l, blocks * 128, n // 16)
    assert int(rows[:, m:].sum()) == 0


def test_rows_beyond_a_tile_width_pick_the_next_width_on_batches(sub, oracle):
    """Padded strides and batches through every width: nothing outside C is written."""
    from nvfp4_gemm_b200.inputs import generate_input
    for m in (16, 32, 33, 64, 65, 128):
        n, k, l = 256, 3072, 2
        a, b, sfa, sfb, sfa_perm, sfb_perm, c = generate_input(m, n, k, l, 5)
        store = torch.full((l * m * (n + 24),), 0x7E01, dtype=torch.int16, device="cuda").view(torch.float16)
        wide = torch.as_strided(store, (m, n, l), (n + 24, 1, m * (n + 24)))
        sub.custom_kernel((a, b, sfa, sfb, sfa_perm, sfb_perm, wide))
        sub.check_status()
        assert "decode" in sub.last_kernel()
        assert_bit_exact(wide.contiguous(), expected_fp16(oracle, (a, b, sfa, sfb, sfa_perm, sfb_perm, c)), what=f"m {m}")
        assert int((store.view(torch.int16) == 0x7E01).sum()) == l * m * 24


# a limit is looked at about every millisecond, so the launch has to last some: K is long
@pytest.mark.parametrize("m,kernel", [(32, "gemm_splitk8_decode_t32"), (128, "gemm_splitk8_decode_t128")])
def test_a_split_that_gives_up_reports_it_and_leaves_together(sub, lib, oracle, m, kernel):
    """With a limit of a nanosecond the ranks' waits run out while operands are still streaming in.  The launch
    ends, the host hears of it, and what runs next is right."""
    from nvfp4_gemm_b200 import _lib
    from nvfp4_gemm_b200.inputs import FP4_DTYPE, SF_DTYPE, generate_input
    n, k = 128, 1 << 25
    codes = lambda rows: torch.full((1, rows, k // 2), 0x02, dtype=torch.uint8, device="cuda").permute(1, 2, 0).view(FP4_DTYPE)  # noqa: E731
    atoms = torch.full((1, 1, k // 64, 32, 4, 4), 0x08, dtype=torch.uint8, device="cuda").permute(3, 4, 1, 5, 2, 0).view(SF_DTYPE)
    c = torch.empty((1, m, n), dtype=torch.float16, device="cuda").permute(1, 2, 0)
    data = (codes(m), codes(n), None, None, atoms, atoms, c)
    small = generate_input(m, 256, 12288, 1, 3)
    torch.cuda.synchronize()
    for _ in range(3):
        prev = lib.nvfp4_set_wait_timeout_ns(1)
        try:
            sub.custom_kernel(data)
        finally:
            lib.nvfp4_set_wait_timeout_ns(prev)
        if torch.cuda.get_device_properties(0).multi_processor_count == 148:
            assert sub.last_kernel() == kernel
        with pytest.raises(_lib.Nvfp4Error) as e:
            sub.check_status()
        assert e.value.code == _lib.NVFP4_ERR_DEVICE_TIMEOUT
        sub.custom_kernel(small)
        sub.check_status()
        assert_bit_exact(small[6], expected_fp16(oracle, small), what="after a launch that gave up")
    sub.custom_kernel(data)
    sub.check_status()
    assert torch.equal(c, torch.full_like(c, k // 2 * 2.0 ** -12))     # 1 * 1 and 0 * 0 in turn, scales 2^-6: exact
