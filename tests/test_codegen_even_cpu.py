"""dp_pair_g, the generated f(r)/r of potentials whose f/r is a polynomial in
r^2 and 1/r^2 (even powers of r; also a logarithm, whose force is -1/r):
present exactly for those, and equal to dp_pair_f(r)/r (both compiled for the
host in double) over the distances a pair loop meets."""
import re
import shutil
import subprocess

import pytest

from dompap_gb300 import codegen

EVEN = ["4*(r**-12-r**-6)", "r**2/2 + 0.1*r**-4", "1-r**2", "2.5*r**4 - 3/r**2", "0*r", "3*(r**-10 - 0.7*r**-2)",
        "r**-64 + 1e-3*r**64",
        "log(r)"]
ODD = ["(1-r)**2", "r**-9 - r**-6", "4*(r**-12-r**-6) + exp(-r)", "r**-12 - (r - 2.5)", "sqrt(r)", "cos(r**2)",
       "r**-130", "1/(1+r**2)", "r*log(r)"]

HARNESS = r"""
#include <cmath>
#include <cstdio>
#define __device__
#define __forceinline__ inline
template <typename R> inline R dp_k(float v) { return R(v); }
%s
int main() {
    double worst = 0.0;
    for (int i = 0; i <= 400; ++i) {
        const double r = 0.7 + 0.007 * i, g = dp_pair_g<double>(r * r, 1.0 / (r * r)), f = dp_pair_f<double>(r, 1.0 / r);
        const double scale = std::fabs(f / r) + std::fabs(g);
        if (scale > 1e-3) worst = std::fmax(worst, std::fabs(g - f / r) / scale);
    }
    std::printf("%%.17g\n", worst);
}
"""


@pytest.mark.parametrize("potential", ODD)
def test_absent_for_other_potentials(potential):
    assert "dp_pair_g" not in codegen.make_pair_source(potential, 2.5)[0]


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
@pytest.mark.parametrize("potential", EVEN)
def test_equals_force_over_r(potential, tmp_path):
    source = codegen.make_pair_source(potential, 2.5)[0]
    assert re.search(r"^#define DP_PAIR_EVEN 1$", source, flags=re.M)
    (tmp_path / "g.cpp").write_text(HARNESS % source)
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", str(tmp_path / "g"), str(tmp_path / "g.cpp")], check=True)
    worst = float(subprocess.run([str(tmp_path / "g")], capture_output=True, text=True, check=True).stdout)
    # up to ~130 roundings of a power against ~65 of the other's, 1.1e-16 each,
    # and cancellation between two terms no worse than 1e3 of their sum
    assert worst <= 1e-11
