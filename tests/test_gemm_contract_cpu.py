"""What the internal products refuse on the host, before anything touches a device."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cuda_ltc_b200")
CUDA_INC = "/usr/local/cuda/include"

SRC = r"""
#include <cstdio>
#include "gemm_fp32.h"
int main() {
    ltca_ctx ctx;
    ctx.sm_count = ctx.sm_device = 148;
    float* p = reinterpret_cast<float*>(256);       // never read
    const ltca::Gemm32Problem g = {p, p, p, p, 64, 64, 65536, 65536, 64, 64};
    const int rc = ltca::gemm_fp32(&ctx, &g, 1, 0, 0, false, true, p, 1 << 24);
    std::printf("%d %s\n", rc, ctx.err);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INC), reason="needs g++ and CUDA headers")
def test_a_sliced_product_with_a_bias_is_refused(tmp_path):
    """The slices' results meet in a second kernel that adds no bias: 64 x 64 from a contraction of 65536 is sliced."""
    from cuda_ltc_b200.build import build_library
    build_library()
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-I", os.path.join(PKG, "csrc"), "-I", CUDA_INC, str(src), "-o", str(exe),
                           f"-L{PKG}", "-l:libltc_attn.so", f"-Wl,-rpath,{PKG}"])
    out = subprocess.check_output([str(exe)], text=True)
    assert out.startswith("-1 ") and "bias" in out, out
