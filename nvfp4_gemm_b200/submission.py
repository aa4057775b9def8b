"""The operator entry point, with the reference's signature (template.py:4-25):

    custom_kernel(data) -> c,   data = (a, b, sfa, sfb, sfa_permuted, sfb_permuted, c)

``c`` is pre-allocated by the caller, written in place and returned (template.py:20).
``b.shape[0] == 1`` selects the GEMV (same tuple positions, old_files/1.py:697-698); every
other shape goes to the tensor-core GEMM, which reads the permuted scale tensors like
s_128t.py:605-609.  The work is enqueued on torch's current CUDA stream and not waited for.
All compute happens in the CUDA library behind the C ABI; there is no PyTorch or CPU path.
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib
from ._lib import GemmConfig, Nvfp4Error, Problem
from .task import input_t, output_t


def _batch_stride(t: torch.Tensor, dim: int = 2) -> int:
    return t.stride(dim) if t.shape[dim] > 1 else 0


def make_problem(data: input_t) -> Problem:
    """Translate the 7-tuple into the C ABI's ``nvfp4_problem`` (pointers, sizes, strides)."""
    p = Problem()
    _lib.native().fill_problem(tuple(data), ctypes.addressof(p))
    return p


def _require_cuda(data: input_t) -> None:
    if not all(t.is_cuda for t in data if t is not None):
        raise ValueError("custom_kernel needs CUDA tensors (there is no CPU fallback)")


def custom_kernel(data: input_t) -> output_t:
    status = _lib.native().matmul(data)
    if status:
        _lib.check(status)
    return data[6]


def gemm(data: input_t, tile_n: int = 0, epilogue: int = 0, grid: int = 0, cta_group: int = 0,
         split_k: int = 0, raster: int = 0) -> output_t:
    """The GEMM with an explicit kernel configuration (tests and tuning)."""
    lib = _lib.load()
    _require_cuda(data)
    problem = make_problem(data)
    cfg = GemmConfig(tile_n, epilogue, grid, cta_group, split_k, raster)
    stream = torch.cuda.current_stream(data[0].device).cuda_stream
    with torch.cuda.device(data[0].device):
        _lib.check(lib.nvfp4_gemm(problem, cfg, stream))
    return data[6]


_ACTIVATIONS = {"none": _lib.ACT_NONE, "relu": _lib.ACT_RELU, "silu": _lib.ACT_SILU}


def gemm_epilogue(data: input_t, bias=None, activation: str = "none", nvfp4_out: bool = False, tile_n: int = 0, grid: int = 0,
                  cta_group: int = 0, split_k: int = 0, out=None):
    """The GEMM with the step that follows it fused into its epilogue: ``act(a @ b.T + bias)``.

    ``nvfp4_out=False`` writes fp16 into ``data[6]`` and returns it.  ``nvfp4_out=True`` returns
    the result re-quantised to NVFP4 as ``(packed, sf, sf_permuted)`` -- [M, N/2, L] packed e2m1,
    [M, N/16, L] e4m3 scales and the same scales in the permuted atom layout -- i.e. the ``a``,
    ``sfa`` and ``sfa_permuted`` of a following ``custom_kernel`` call whose K is this N; ``data[6]``
    may then be None; ``out`` may pass the triple a previous call returned, to be overwritten
    instead of allocating a new one.  The reference writes fp16 only (sub_cub.py:98-104); no
    counterpart."""
    if not nvfp4_out:
        out = None
    elif out is None:
        out = _empty_nvfp4(data[0].shape[0], data[1].shape[0], data[0].shape[2], data[0].device)
    _lib.check(_lib.native().gemm_epilogue(data, bias, _ACTIVATIONS[activation], out, tile_n, grid, cta_group, split_k))
    return out if nvfp4_out else data[6]


def _empty_nvfp4(m: int, n: int, l: int, device):
    """Memory for an [m, n, l] result in NVFP4: packed codes, plain scales, permuted scales."""
    from .inputs import FP4_DTYPE, SF_DTYPE
    packed = torch.empty((l, m, n // 2), dtype=torch.uint8, device=device)
    sf = torch.empty((l, m, n // 16), dtype=torch.uint8, device=device)
    sf_perm = torch.empty((l, (m + 127) // 128, n // 64, 32, 4, 4), dtype=torch.uint8, device=device)
    return (packed.permute(1, 2, 0).view(FP4_DTYPE), sf.permute(1, 2, 0).view(SF_DTYPE),
            sf_perm.permute(3, 4, 1, 5, 2, 0).view(SF_DTYPE))


def check_scale_layouts(data: input_t) -> None:
    """Validate that the plain and the permuted scale tensors of one operator call say the same
    (the harness passes both, template.py:11-14; the GEMM reads the permuted ones, the GEMV the
    plain ones).  Compared on the device by ``nvfp4_compare_scale_layouts``; synchronises the
    current stream and raises ValueError naming the first differing scale."""
    a, b, sfa, sfb, sfa_perm, sfb_perm, _ = data
    _require_cuda(data)
    lib = _lib.load()
    k = 2 * a.shape[1]
    stream = torch.cuda.current_stream(a.device).cuda_stream
    result = torch.empty((2, 2), dtype=torch.int64, device=a.device)
    for i, (name, plain, perm, rows) in enumerate((("sfa", sfa, sfa_perm, a.shape[0]), ("sfb", sfb, sfb_perm, b.shape[0]))):
        if perm is None:
            raise ValueError(f"{name}_permuted is missing")
        _lib.check(lib.nvfp4_compare_scale_layouts(plain.data_ptr(), perm.data_ptr(), rows, k, a.shape[2],
                                                   plain.stride(0) if rows > 1 else k // 16, _batch_stride(plain),
                                                   _batch_stride(perm, 5), result[i].data_ptr(), stream))
    counts = result.cpu()
    for i, (name, rows) in enumerate((("sfa", a.shape[0]), ("sfb", b.shape[0]))):
        bad, first = int(counts[i, 0]), int(counts[i, 1])
        if bad:
            col = first % (k // 16)
            row = (first // (k // 16)) % rows
            batch = first // (k // 16) // rows
            raise ValueError(f"{name} and {name}_permuted differ in {bad} scale(s); first at row {row}, scale column {col}, batch {batch}")


def release_stream(stream=None) -> None:
    """Give back the scratch set the GEMM keeps for ``stream`` (default: the current stream), once
    none of its GEMMs is in flight and no graph captured on it will be replayed again."""
    lib = _lib.load()
    stream = stream if stream is not None else torch.cuda.current_stream()
    _lib.check(lib.nvfp4_release_stream(stream.cuda_stream))


def check_status() -> None:
    """Synchronise the current stream and raise if a kernel reported a timed-out wait."""
    lib = _lib.load()
    _lib.check(lib.nvfp4_check_status(torch.cuda.current_stream().cuda_stream))


def last_kernel() -> str:
    return _lib.load().nvfp4_last_kernel().decode()


def launch_count() -> int:
    return int(_lib.load().nvfp4_launch_count())


__all__ = ["custom_kernel", "gemm", "check_status", "last_kernel", "launch_count", "make_problem", "Nvfp4Error"]
