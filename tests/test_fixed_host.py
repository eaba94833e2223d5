"""The integer arithmetic of the FP64 kernels, compiled for the host (no GPU needed)."""
import os
import subprocess
import sys
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "gpu-swimmers_gb300")

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include "fixed_site.cuh"
int main() {
  double x;
  int k;
  while (std::scanf("%la %d", &x, &k) == 2) {
    long long v = 0;
    const bool fits = lbswim::value_to_fixed(x, k, v);
    std::printf("%d %lld\n", fits ? 1 : 0, v);
  }
}
"""


@pytest.fixture(scope="module")
def host_program(tmp_path_factory):
    sys.path.insert(0, PKG)
    import build
    nvcc = build._nvcc()
    d = tmp_path_factory.mktemp("fixed")
    src, exe = d / "fixed.cu", d / "fixed"
    src.write_text(PROGRAM)
    try:
        r = subprocess.run([nvcc, *build.ARCH, "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-I",
                            os.path.join(ROOT, "include"), "-I", build.CSRC, str(src), "-o",
                            str(exe)], capture_output=True, text=True)
    except FileNotFoundError:
        pytest.skip("no nvcc")
    assert r.returncode == 0, r.stderr
    return str(exe)


def test_forces_are_rounded_to_nearest(host_program):
    """A force in the units of a site, 2^(k - 1082): the nearest integer, as near to it from
    below as from above."""
    rng = np.random.default_rng(1)
    k = rng.integers(900, 1150, 4000)
    x = rng.uniform(-1, 1, 4000) * 2.0 ** (k - 1023.0 - rng.integers(4, 70, 4000))
    x[::50] = 2.0 ** (k[::50] - 1083.0)          # half a unit
    x[1::50] = -np.nextafter(2.0 ** (k[1::50] - 1083.0), 0)
    x[2::50] = 0.0
    x[3::50] = 2.0 ** -1070
    lines = "".join("%s %d\n" % (float(a).hex(), b) for a, b in zip(x, k))
    out = subprocess.run([host_program], input=lines, capture_output=True, text=True, check=True)
    got = [tuple(map(int, ln.split())) for ln in out.stdout.split("\n") if ln]
    assert len(got) == len(x)
    off = []
    for i, (a, b, (fits, v)) in enumerate(zip(x, k, got)):
        want = Fraction(float(a)) / Fraction(2) ** (int(b) - 1082)
        assert fits == (abs(want) < 2 ** 56)
        if fits:
            assert abs(v - want) <= Fraction(1, 2)
            if i % 50 > 3:
                off.append(float(v - want))
    # the mean of 3800 values of at most a half: five standard errors
    assert abs(np.mean(off)) < 5 * 0.5 / np.sqrt(3 * 3800)
