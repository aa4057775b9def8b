"""The decode kernel's epilogue beside bias, ReLU and dense outputs, and its sums on scales of every size."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sub(lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nvfp4_gemm_b200 import submission
    return submission


# one shape per tile width with and without a split of K, rows short of the tile
EPILOGUE_SHAPES = [(17, 384, 1792, 2), (31, 2560, 3072, 1), (7, 128, 2048, 3), (63, 256, 1024, 1), (64, 256, 2304, 2), (40, 6400, 512, 3),
                   (97, 256, 3328, 2), (127, 128, 12288, 1), (300, 384, 3072, 2)]


def _bias(n):
    return (torch.randn(n, generator=torch.Generator().manual_seed(4)) * 64).half().cuda()


@pytest.mark.parametrize("shape", EPILOGUE_SHAPES)
@pytest.mark.parametrize("nvfp4_out", [False, True])
@pytest.mark.parametrize("activation", ["none", "silu"])
def test_decode_epilogue_activations_equal_the_persistent_kernels(sub, shape, nvfp4_out, activation):
    """The sums are exact in any order and the epilogues do the same to them, so the bytes are equal."""
    from nvfp4_gemm_b200.inputs import generate_input
    data = generate_input(*shape, 80)
    bias = _bias(shape[1])
    got = []
    for kw in ({}, {"split_k": 1}):
        data[6].view(torch.int16).fill_(0x7fff)
        out = sub.gemm_epilogue(data, bias=bias, activation=activation, nvfp4_out=nvfp4_out, **kw)
        sub.check_status()
        assert ("decode" in sub.last_kernel()) == (not kw)
        got.append([t.view(torch.uint8).clone() for t in out] if nvfp4_out else [out.view(torch.int16).clone()])
    for g, e in zip(*got):
        assert torch.equal(g, e)


@pytest.mark.parametrize("shape", EPILOGUE_SHAPES)
@pytest.mark.parametrize("left_out", [None, "out_sf", "out_sf_perm"])
def test_decode_epilogue_writes_what_is_asked_for_at_padded_strides(sub, lib, shape, left_out):
    """Rows, batches and scale blocks further apart than they have to be, and either scale layout left out:
    the values are those of the dense call, and nothing between them is written."""
    from nvfp4_gemm_b200 import _lib
    from nvfp4_gemm_b200.inputs import generate_input
    m, n, k, l = shape
    data = generate_input(*shape, 81)[:6] + (None,)
    bias = _bias(n)
    packed, sf, sf_perm = sub.gemm_epilogue(data, bias=bias, activation="relu", nvfp4_out=True, split_k=1)
    blocks, row_bytes = (m + 127) // 128, n // 64 * 512
    pads = {"out_packed": (m + 1, n // 2 + 16, n // 2), "out_sf": (m + 1, n // 16 + 2, n // 16), "out_sf_perm": (blocks + 1, row_bytes + 16, row_bytes)}
    store = {name: torch.full((l, rows, stride), 0xA5, dtype=torch.uint8, device="cuda") for name, (rows, stride, _) in pads.items()}
    e = _lib.Epilogue()
    e.bias, e.activation, e.output = bias.data_ptr(), _lib.ACT_RELU, _lib.OUT_NVFP4
    for name, (rows, stride, _) in pads.items():
        if name != left_out:
            setattr(e, name, store[name].data_ptr())
        setattr(e, name + ("_block_stride" if name == "out_sf_perm" else "_row_stride"), stride)
        setattr(e, name + "_batch_stride", rows * stride)
    _lib.check(lib.nvfp4_gemm_epilogue(sub.make_problem(data), None, e, torch.cuda.current_stream().cuda_stream))
    sub.check_status()
    assert "decode" in sub.last_kernel()
    exp = {"out_packed": packed.view(torch.uint8).permute(2, 0, 1), "out_sf": sf.view(torch.uint8).permute(2, 0, 1),
           "out_sf_perm": torch.as_strided(sf_perm.view(torch.uint8), (l, blocks, row_bytes), (blocks * row_bytes, row_bytes, 1))}
    for name, (rows, stride, used) in pads.items():
        canary = store[name].clone()
        if name != left_out:
            assert torch.equal(store[name][:, :rows - 1, :used], exp[name]), name
            canary[:, :rows - 1, :used] = 0xA5
        assert int((canary != 0xA5).sum()) == 0, name


@pytest.mark.parametrize("shape", [(17, 384, 1792, 2), (31, 2560, 3072, 1), (7, 128, 2048, 3), (32, 256, 12288, 1), (50, 128, 12800, 1),
                                   (97, 256, 3328, 2), (300, 384, 3072, 2), (127, 128, 12288, 1)])
def test_decode_general_scales_within_the_rounding_of_their_sums(sub, oracle, shape):
    """Scales of every size: the sums are no longer exact.  Each of the K / 64 additions to an accumulator, and of
    those of the ranks (fewer than 8), may be off by one unit in the last place of the sum of all
    magnitudes; then the result is rounded to fp16."""
    from nvfp4_gemm_b200.inputs import SF_DTYPE, generate_input, permute_scale_factors
    m, n, k, l = shape
    data = list(generate_input(*shape, 82))
    g = torch.Generator().manual_seed(83)
    for i, rows in ((0, m), (1, n)):
        plain = torch.randint(0x20, 0x48, (l, rows, k // 16), dtype=torch.uint8, generator=g).cuda()
        data[2 + i] = plain.permute(1, 2, 0).view(SF_DTYPE)
        data[4 + i] = permute_scale_factors(plain).view(SF_DTYPE)
    out = sub.custom_kernel(tuple(data))
    sub.check_status()
    assert "decode" in sub.last_kernel()
    a, b, sfa, sfb = oracle.tensors_to_numpy(tuple(data))
    got = out.double().cpu().numpy()
    for i in range(l):
        x, y = (oracle.dequantize(v[:, :, i], s[:, :, i]).astype(np.float64) for v, s in ((a, sfa), (b, sfb)))
        exp, magnitude = x @ y.T, np.abs(x) @ np.abs(y).T
        assert np.abs(exp).max() < 60000                     # (no overflow to infinity here)
        assert (np.abs(got[:, :, i] - exp) <= (k / 64 + 8) * 2.0 ** -23 * magnitude + 2.0 ** -11 * np.abs(exp) + 2.0 ** -25).all(), sub.last_kernel()
