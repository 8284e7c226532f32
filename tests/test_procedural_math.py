"""The arithmetic of the two-phase regeneration (procedural.cuh) against the library's own (genn_b200_rng.h, whose division and root
are the correctly rounded ones): the same bits for every one of the 2^23 uniforms, so that regenerated weights and gaps are
those that the initialisation kernels store."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <cuda_runtime.h>
#include "procedural.cuh"
using namespace b200;
enum { UNIFORM, LOGARITHM, QUOTIENT, ROOT, COSINE, NORMAL, CHECKS };
__global__ void compareKernel(unsigned int *differ)
{
    const unsigned int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= (1u << 23)) return;
    auto check = [&](int what, float a, float b) { if(__float_as_uint(a) != __float_as_uint(b)) atomicAdd(&differ[what], 1u); };
    // (the low nine bits of a random word are dropped)
    const unsigned int x = (i << 9) | (i & 511u);
    const float u = b200_u32_to_uniform(x), l = b200_logf(u);
    check(UNIFORM, proceduralUniform(x), u);
    check(LOGARITHM, proceduralLog(u), l);
    const float y = -2.0f * l;
    check(ROOT, proceduralRoot(y), __fsqrt_rn(y));
    float s, c;
    b200_sincos2pif(u, &s, &c);
    check(COSINE, proceduralCos(u), c);
    check(NORMAL, B200_FMUL(proceduralRoot(B200_FMUL(-2.0f, proceduralLog(u))), proceduralCos(proceduralUniform(~x))),
          [&] { b200_sincos2pif(b200_u32_to_uniform(~x), &s, &c); return B200_FMUL(__fsqrt_rn(B200_FMUL(-2.0f, l)), c); }());
    // the corrected quotient on its own, over every mantissa the logarithm divides by
    const float m = __uint_as_float(0x3F3504F4u + i), n = m - 1.0f, d = m + 1.0f;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = __fmul_rn(n, r);
    check(QUOTIENT, __fmaf_rn(__fmaf_rn(-d, q, n), r, q), __fdiv_rn(n, d));
}
int main()
{
    unsigned int *differ, host[CHECKS];
    if(cudaMalloc(&differ, sizeof(host)) || cudaMemset(differ, 0, sizeof(host))) return 1;
    compareKernel<<<(1u << 23) / 256u, 256>>>(differ);
    if(cudaMemcpy(host, differ, sizeof(host), cudaMemcpyDeviceToHost)) return 2;
    for(int i = 0; i < CHECKS; i++) printf("%u ", host[i]);
    return 0;
}
"""


@pytest.mark.gpu
def test_every_uniform_gives_the_bits_of_the_library(tmp_path):
    nvcc = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    (tmp_path / "compare.cu").write_text(SOURCE)
    exe = str(tmp_path / "compare")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-diag-suppress", "186,177", "-I",
                           os.path.join(REPO, "genn_b200", "csrc"), "-I", os.path.join(REPO, "include"), str(tmp_path / "compare.cu"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0
    assert out.stdout.split() == ["0"] * 6, "uniform, logarithm, quotient, root, cosine, normal: " + out.stdout
