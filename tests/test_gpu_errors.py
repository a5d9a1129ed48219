"""Rounding errors of FP64 kernels against 80-bit sums (tests/kernel_errors.cu):
the reciprocal square roots against their bounds, the 8x8 Hadamard and the
separable transforms against the error of the same sums done plainly in FP64
on the host (a tenth more, which is what two equally exact orders of sums
differ by over these few thousand outputs)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "exafmm-rd_b200")


@pytest.fixture(scope="module")
def errors(pkg, tmp_path_factory):
    pkg.rtfmm.lib()  # the library is built
    exe = str(tmp_path_factory.mktemp("errors") / "kernel_errors")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(PKG, "csrc"), os.path.join(ROOT, "tests", "kernel_errors.cu"), "-o", exe, "-L", PKG,
                    "-lrtfmm_b200", "-Xlinker", "-rpath," + PKG, "-Xcompiler", "-fopenmp"], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    print(out.stdout)
    assert out.returncode == 0, out.stdout + out.stderr
    return {name: (float(e), float(bound)) for name, e, bound in (line.split() for line in out.stdout.splitlines())}


@pytest.mark.parametrize("check", ["rsqrt", "rsqrt_twice", "rsqrt_zero", "hadamard", "hadamard_heavy"] +
                         ["%s_%d%s" % (d, P, s) for d in ("up", "down") for P in range(4, 11) for s in ("", "_smooth")])
def test_error(errors, check):
    e, bound = errors[check]
    assert e <= bound
