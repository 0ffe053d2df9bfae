"""The pair passes' square root and reciprocal (the hardware approximation with one
Newton-Raphson step) against 64 bits: the step leaves the error below one unit in the last
place (the approximations' own bounds are 2 and 1 ulp)."""
import subprocess
from pathlib import Path

import pytest

from warpsph_b200 import build

pytestmark = pytest.mark.gpu


def test_newton_step_is_within_one_ulp(cuda, tmp_path):
    src = Path(__file__).resolve().parent / "native" / "newton_check.cu"
    exe = tmp_path / "newton_check"
    subprocess.run([build.nvcc(), *build.ARCH_FLAGS, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.INCLUDE), "-I",
                    str(build.CSRC), str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert float(out[1]) <= 1.0 and float(out[3]) <= 1.0, out
    assert float(out[5]) == 0.0, out


def test_markstein_quotients_are_rounded(cuda, tmp_path):
    """The reciprocal over every significand but the all-ones one, and 76 million quotients, equal
    those of the rounded division."""
    src = Path(__file__).resolve().parent / "native" / "div_check.cu"
    exe = tmp_path / "div_check"
    subprocess.run([build.nvcc(), *build.ARCH_FLAGS, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.INCLUDE), "-I",
                    str(build.CSRC), str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["rcp", "0", "div", "0", "div2", "0"], out


def test_newton_bounds_hold_up_to_the_ends_of_the_range(cuda, tmp_path):
    """Every exponent from the subnormals up, zeros, infinities and NaN: zero results outside the
    stated bounds (a reciprocal of 0 is infinite and of an infinity 0, as the division's)."""
    src = Path(__file__).resolve().parent / "native" / "newton_domain_check.cu"
    exe = tmp_path / "newton_domain_check"
    subprocess.run([build.nvcc(), *build.ARCH_FLAGS, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.INCLUDE), "-I",
                    str(build.CSRC), str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["sqrt", "0", "rcp", "0", "special", "0"], out


def test_pair_image_equals_the_conditional_shift(cuda, tmp_path):
    """The minimum image of the pair sums, bit for bit, around half the box above all."""
    here = Path(__file__).resolve().parent / "native"
    exe = tmp_path / "image_check"
    subprocess.run([build.nvcc(), *build.ARCH_FLAGS, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.INCLUDE), "-I",
                    str(build.CSRC), str(here / "image_check.cu"), str(build.CSRC / "sph_neighbors.cu"), "-o", str(exe)], check=True,
                   capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out[:3] == ["differ", "0", "of"] and int(out[3]) > 900000, out
