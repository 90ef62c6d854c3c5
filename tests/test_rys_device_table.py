"""The device form of the Rys rule's table (rys_rule.h: rys_device_table,
powers of the interval's coordinate, roots side by side) against the host
rule rys_rule evaluates, at the degrees the kernels read: FP64 to two units in
the last place of the host's own Clenshaw sum, FP32 to FP32 accuracy."""

import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "felizjueves_b200", "csrc")

SRC = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include "rys_rule.h"
using namespace fjb;
template <typename R>
static double worst(int deg, const std::vector<double> &host) {
    const std::vector<double> d = rys_device_table(deg);
    const std::vector<R> t(d.begin(), d.end());
    double e = 0.0;
    for (int n = 1; n <= kRysMaxN; ++n)
        for (int i = 0; i <= 4 * kRysNI; ++i) {  // interval edges and insides, and past the switch
            const double T = i / 4.0 + (i % 3) * 0.03125;
            double x[kRysMaxN], w[kRysMaxN];
            rys_rule(n, T, host.data(), x, w);
            for (int r = 0; r < n; ++r) {
                double v[2];
                if (T < kRysTSwitch) {
                    const int k0 = std::min((int)T, kRysNI - 1);
                    const R u = (R)(2.0 * (T - k0) - 1.0);
                    for (int c = 0; c < 2; ++c) {
                        R p = t[rys_device_at(deg, n, k0, deg, r) + c];
                        for (int k = deg - 1; k >= 0; --k) p = std::fma(p, u, t[rys_device_at(deg, n, k0, k, r) + c]);
                        v[c] = p;
                    }
                } else {
                    v[0] = t[rys_device_asym(deg, n) + 2 * r] / T;
                    v[1] = t[rys_device_asym(deg, n) + 2 * r + 1] * (0.5 / std::sqrt(T));
                }
                e = std::max({e, std::fabs(v[0] / x[r] - 1.0), std::fabs(v[1] / w[r] - 1.0)});
            }
        }
    return e;
}
int main() {
    const std::vector<double> host = rys_table();
    std::printf("%.3e %.3e\n", worst<double>(kRysDegD, host), worst<float>(kRysDegF, host));
}
"""


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    d = tmp_path_factory.mktemp("rysdev")
    (d / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-I", CSRC, str(d / "t.cpp"),
                    os.path.join(CSRC, "rys_table.cpp"), "-o", str(d / "t")], check=True)
    return tuple(map(float, subprocess.run([str(d / "t")], check=True, capture_output=True, text=True).stdout.split()))


def test_device_rule_matches_host_rule(errors):
    # two roundings apart on each side (coefficient, last sum): 4 x 1.1e-16,
    # and the same in FP32, 4 x 6e-8
    assert errors[0] <= 4.5e-16
    assert errors[1] <= 2.4e-7
