"""rcp_screened (csrc/xpr_math.cuh): one Newton step on the hardware's reciprocal gives the
correctly rounded one.  On the CPU from every approximation that the instruction's documented
error (one ulp) allows; on the GPU against __frcp_rn."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "xpulse_recon_b200", "csrc")

CPU = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
static float f_of(uint32_t u) { float x; memcpy(&x, &u, 4); return x; }
static uint32_t u_of(float x) { uint32_t u; memcpy(&u, &x, 4); return u; }
int main(void)
{
    long checked = 0, wrong = 0, wrong_ones = 0;
    for (uint32_t m = 0; m < 1u << 23; ++m) {
        const float b = f_of(0x3f800000u | m), exact = 1.0f / b;
        for (int d = -2; d <= 2; ++d) {
            const float y = f_of(u_of(exact) + (uint32_t)d);
            if (fabs((double)y - 1.0 / (double)b) > (y < 1.0f ? 0x1p-24 : 0x1p-23)) continue;
            ++checked;
            if (fmaf(fmaf(-b, y, 1.0f), y, y) != exact) m == 0x7fffffu ? ++wrong_ones : ++wrong;
        }
    }
    printf("%ld %ld %ld\n", checked, wrong, wrong_ones);
    return 0;
}
"""

GPU = r"""
#include <cstdio>
#include "xpr_math.cuh"
__global__ void check(uint32_t sign_exp, unsigned *wrong)
{
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;  // 2^23 threads
    const float b = __uint_as_float(sign_exp << 23 | m);
    if (__float_as_uint(xpr::rcp_screened(b)) != __float_as_uint(__frcp_rn(b))) atomicAdd(wrong, 1u);
}
int main()
{
    unsigned *wrong;
    if (cudaMallocManaged(&wrong, 4) != cudaSuccess) return 2;
    *wrong = 0;
    for (uint32_t e : {127u - 60u, 126u, 127u, 128u, 127u + 59u, 256u + 127u, 256u + 127u - 59u})
        check<<<(1 << 23) / 256, 256>>>(e, wrong);
    if (cudaDeviceSynchronize() != cudaSuccess) return 3;
    printf("%u\n", *wrong);
    return 0;
}
"""


def test_one_newton_step_from_any_approximation(tmp_path):
    if shutil.which("gcc") is None:
        pytest.skip("no gcc")
    src, exe = tmp_path / "r.c", tmp_path / "r"
    src.write_text(CPU)
    subprocess.run(["gcc", "-O2", "-mfma", "-ffp-contract=off", str(src), "-o", str(exe), "-lm"], check=True)
    checked, wrong, wrong_ones = (int(x) for x in subprocess.check_output([str(exe)]).split())
    assert checked >= 2 ** 24 - 1 and wrong == 0
    assert wrong_ones == 1  # the mantissa of all ones, from the float below


@pytest.mark.gpu
def test_every_mantissa_against_the_device(tmp_path):
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc")
    src, exe = tmp_path / "r.cu", tmp_path / "r"
    src.write_text(GPU)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--fmad=false", "-I", CSRC,
                    str(src), "-o", str(exe)], check=True)
    assert int(subprocess.check_output([str(exe)])) == 0
