"""Which SGEMMs the host rule sends to the tensor cores, at measured shapes
on 152 SMs (CPU: a host function of the library)."""
import ctypes as C

import pytest


@pytest.mark.parametrize("m,n,k,tensor", [
    (1, 1, 1, 0), (64, 64, 64, 0), (128, 128, 128, 0), (300, 300, 300, 0), (32, 4096, 256, 0), (1000, 48, 48, 0),
    (1, 1, 1 << 20, 0), (2000, 2000, 7, 0), (64, 64, 1024, 1), (384, 384, 384, 1), (100, 3000, 200, 1),
    (1024, 1024, 16, 1), (2000, 2000, 8, 1), (8, 4096, 4096, 1), (4096, 4096, 4096, 1),
    (0x7fffffff, 0x7fffffff, 0x7fffffff, 1)])
def test_choice(m, n, k, tensor):
    import libgpublas_gb300 as g
    lib = g.load()
    lib.gbx_sgemm_tensor_choice.argtypes = [C.c_int] * 4
    assert lib.gbx_sgemm_tensor_choice(m, n, k, 152) == tensor
