"""The tiled passes take PTX's ex2.approx.ftz where the direct ones call exp2f: the two give
the same bits for every FP32 exponent from -126, below which results are subnormal, to 0."""
import ctypes as C
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cuda_runtime.h>
__global__ void compare(unsigned first, unsigned last, unsigned long long *differ) {
    for (unsigned long long b = first + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; b <= last;
         b += (unsigned long long)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((unsigned)b);
        float y;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
        if (__float_as_uint(y) != __float_as_uint(exp2f(x))) atomicAdd(differ, 1ull);
    }
}
extern "C" int run(unsigned first, unsigned last, unsigned long long *differ) {
    compare<<<1024, 256>>>(first, last, differ);
    return (int)cudaDeviceSynchronize();
}
"""


def test_exponentials_agree(tmp_path, cuda):
    import torch

    from apbf_gb300 import build as b

    (tmp_path / "ex2.cu").write_text(SOURCE)
    so = tmp_path / "ex2.so"
    subprocess.run([b.nvcc(), *b.ARCH, *b.COMMON, "-shared", "-o", str(so), str(tmp_path / "ex2.cu")], check=True)
    differ = torch.zeros(1, dtype=torch.int64, device=cuda)
    first, last = 0x80000000, 0xC2FC0000  # -0 to -126
    assert C.CDLL(str(so)).run(C.c_uint(first), C.c_uint(last), C.c_void_p(differ.data_ptr())) == 0
    assert int(differ.item()) == 0
