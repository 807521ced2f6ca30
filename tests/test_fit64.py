"""The polynomials of the FP64 pair factor (csrc/p2p_fit64.h), compiled for the
host and evaluated as the kernel does, against long double."""
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "p2p_fit64.h"
using namespace p2p;
int main(int argc, char **argv) {
    const double xc = atof(argv[1]), rs = atof(argv[2]), k = 0.5 / rs;
    const Fit64 F = fit64(xc, rs, 1e-6 * rs);
    double worst = 0;
    for (int i = 0; F.nfar && i < 200000; ++i) {
        const double x = xc * (i + 0.5) / 200000 * (1 - 1e-9), r2 = (x / k) * (x / k);
        const long double R = sqrtl(r2), X = R * 0.5L / rs;
        const long double want = (erfcl(X) + 2 / sqrtl(kFit64Pi) * X * expl(-X * X)) / (R * R * R);
        const double y = (double)(1 / R);
        double f;
        if (fit64_hi(r2) < F.hi_near) {
            f = F.near[kFit64Near - 1];
            for (int c = kFit64Near - 2; c >= 0; --c) f = fma(f, r2 - F.near_mid, F.near[c]);
            f = fma(y * y, y, f);
        } else {
            const double n = rint(r2 * F.e_hi), t = fma(r2, F.e_lo, fma(r2, F.e_hi, -n)), s = fma(r2, y, -F.far_mid);
            double e = F.exp2[kFit64Exp - 1], q = F.far[F.nfar - 1];
            for (int c = kFit64Exp - 2; c >= 0; --c) e = fma(e, t, F.exp2[c]);
            for (int c = F.nfar - 2; c >= 0; --c) q = fma(q, s, F.far[c]);
            f = y * y * y * (ldexp(e, (int)n) * q);
        }
        worst = fmax(worst, fabs((double)((f - want) / want)));
    }
    printf("%d %.6e\n", F.nfar, worst);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("fit64")
    (d / "f.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-march=x86-64-v3", "-I",
                           os.path.join(REPO, "photons-on-mt3000_b200", "csrc"), str(d / "f.cpp"), "-o", str(d / "f")])
    return str(d / "f")


@pytest.mark.parametrize("x_cut,coefs", [(1.25, 17), (2.25, 17), (2.8125, 19), (3.5, 22), (4.0, 25)])
@pytest.mark.parametrize("rs", [0.0046875, 1.7, 3e4])
def test_pair_factor_is_within_ten_half_ulps(program, x_cut, coefs, rs):
    """y^3 costs up to 4 roundings of y and 2 products, near pairs lose up to
    1 / 0.55 of that; 1e-15 is nine half units in the last place."""
    n, err = subprocess.check_output([program, str(x_cut), str(rs)], text=True).split()
    assert int(n) == coefs
    assert float(err) <= 1.0e-15


@pytest.mark.parametrize("x_cut", [0.0, -1.0, 1.0, 4.5, float("nan")])
def test_other_cutoffs_have_no_fit(program, x_cut):
    assert subprocess.check_output([program, str(x_cut), "0.1"], text=True).split()[0] == "0"


KEPT = r"""
#include <cstdio>
#include <cstdlib>
#include "p2p_fit64.h"
using namespace p2p;
static bool same(const Fit64 &a, const Fit64 &b) {
    bool s = a.nfar == b.nfar && a.hi_near == b.hi_near && a.hi_in == b.hi_in && a.hi_out == b.hi_out &&
             a.near_mid == b.near_mid && a.far_mid == b.far_mid && a.e_hi == b.e_hi && a.e_lo == b.e_lo;
    for (int i = 0; i < kFit64Near; ++i) s = s && a.near[i] == b.near[i];
    for (int i = 0; i < kFit64MaxFar; ++i) s = s && a.far[i] == b.far[i];
    for (int i = 0; i < kFit64Exp; ++i) s = s && a.exp2[i] == b.exp2[i];
    return s;
}
int main() {
    // x_cut, split radius, softening, and whether the fit has to be made
    const double call[][4] = {{2.8125, 0.01, 1e-4, 1}, {2.8125, 0.01, 1e-4, 0}, {2.25, 0.01, 1e-4, 1}, {2.25, 0.02, 1e-4, 1},
                              {2.25, 0.02, 1e-70, 1}, {2.25, 0.02, 1e-70, 0}, {2.25, 0.02, 1e-4, 1}, {0.0, 0.02, 1e-4, 1},
                              {0.0, 0.02, 1e-4, 0}, {2.8125, 0.01, 1e-4, 1}};
    Fit64For kept;
    int wrong = kept.fit().nfar != 0;
    for (auto &c : call) {
        if (kept.set(c[0], c[1], c[2]) != (c[3] != 0)) ++wrong;
        if (!same(kept.fit(), fit64(c[0], c[1], c[2]))) ++wrong;
    }
    printf("%d\n", wrong);
}
"""


def test_the_fit_is_made_again_only_for_other_numbers(tmp_path):
    (tmp_path / "k.cpp").write_text(KEPT)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", os.path.join(REPO, "photons-on-mt3000_b200", "csrc"),
                           str(tmp_path / "k.cpp"), "-o", str(tmp_path / "k")])
    assert subprocess.check_output([str(tmp_path / "k")], text=True).split() == ["0"]
