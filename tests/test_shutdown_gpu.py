"""The library after nvfp4_shutdown() and a reset of the process's own context."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu

# torch holds no memory here: it would go with the context
_SCRIPT = """
import ctypes
import sys
from cuda.bindings import runtime as rt
from nvfp4_gemm_b200 import _lib

lib = _lib.load()

def ok(r):
    assert int(r[0]) == 0, r
    return r[1] if len(r) == 2 else None

def product(m, n, k):
    p = _lib.Problem()
    p.m, p.n, p.k, p.l = m, n, k, 1
    for name, size, byte in (("a", m * k // 2, 0x22), ("b", n * k // 2, 0x22), ("sfa_perm", 128 * k // 16, 0x38), ("sfb_perm", n * k // 16, 0x38), ("c", 2 * m * n, 0xFF)):
        ptr = ok(rt.cudaMalloc(size))
        ok(rt.cudaMemset(ptr, byte, size))
        setattr(p, name, ptr)
    p.a_row_stride = p.b_row_stride = k // 2
    p.c_row_stride = n
    _lib.check(lib.nvfp4_matmul(p, None))
    _lib.check(lib.nvfp4_check_status(None))
    out = (ctypes.c_uint16 * (m * n))()
    ok(rt.cudaMemcpy(ctypes.addressof(out), p.c, 2 * m * n, rt.cudaMemcpyKind.cudaMemcpyDeviceToHost))
    return lib.nvfp4_last_kernel().decode(), set(out)

shapes = [(20, 256, 512), (60, 256, 512), (100, 256, 4096), (256, 256, 256)]
before = [product(*s) for s in shapes]
lib.nvfp4_shutdown()
ok(rt.cudaDeviceReset())
assert [product(*s) for s in shapes] == before
for (name, values), s in zip(before, shapes):
    assert values == {{512: 0x6000, 4096: 0x6C00, 256: 0x5C00}[s[2]]}, (s, name, values)     # fp16 512, 4096, 256
print("same", *(name for name, _ in before))
"""


def test_kernels_launch_again_after_shutdown_and_a_new_context(lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, "-c", _SCRIPT], cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.startswith("same") and r.stdout.count("decode") == 3
