"""The FP32 bound on the walk's pair test (csrc/p2p_walk_test.h), compiled for the
host, against the test in FP64: where it decides, it decides the same."""
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "p2p_walk_test.h"
using namespace p2p;
static int exact(const WalkBox &i, const WalkBox &j, bool an, bool bn, double cutoff, double angle) {
    double dist[3], w[3], mn[3];
    for (int d = 0; d < 3; ++d) {
        dist[d] = i.c[d] - j.c[d];
        w[d] = (i.w[d] + j.w[d]) * 0.5;
        const double m = std::fabs(dist[d]) - w[d];
        mn[d] = m <= 0.0 ? 0.0 : m;
    }
    const double dd2 = dist[0] * dist[0] + dist[1] * dist[1] + dist[2] * dist[2];
    int t = 0;
    if (!(mn[0] + mn[1] + mn[2] < 1.0e-15)) {
        const double dm2 = mn[0] * mn[0] + mn[1] * mn[1] + mn[2] * mn[2];
        const double wm = 2.0 * std::fabs(std::max(w[0], std::max(w[1], w[2])));
        if (dm2 > cutoff * cutoff) return WALK_DROP;
        if (wm * wm < angle * angle * dd2) t = 1;
    }
    if (t) return WALK_ACCEPT;
    return an && (!bn || i.sum > j.sum) ? WALK_OPEN_A : WALK_OPEN_B;
}
int main(int argc, char **argv) {
    const double box = atof(argv[1]), angle = atof(argv[2]), offset = atof(argv[3]);
    std::mt19937_64 g(5);
    std::uniform_real_distribution<double> u(0, 1);
    long wrong = 0, decided = 0, n = 400000;
    for (long q = 0; q < n; ++q) {
        const double cutoff = box * (q % 7 ? 0.02 : 0.0);
        WalkBox a, b;
        WalkBox32 fa, fb;
        // gaps from touching to a few cutoffs, widths over six decades, some pairs
        // placed on the boundaries of the test
        for (int d = 0; d < 3; ++d) {
            a.w[d] = box * std::pow(10.0, -1 - 5 * u(g));
            b.w[d] = q % 3 ? a.w[d] * (0.5 + u(g)) : box * std::pow(10.0, -1 - 5 * u(g));
            if (q % 11 == 0) b.w[d] = a.w[d];
            a.c[d] = offset + box * u(g);
            double gap = cutoff * std::pow(10.0, 1 - 4 * u(g));
            if (q % 5 == 0) gap = d ? -1e-3 * box : cutoff * (1 + (u(g) - 0.5) * std::pow(10.0, -16 * u(g)));
            if (q % 13 == 0) gap = 0;
            b.c[d] = a.c[d] + (u(g) < 0.5 ? -1 : 1) * (gap + 0.5 * (a.w[d] + b.w[d]));
        }
        if (angle > 0 && q % 17 == 0) {  // on the acceptance boundary along x
            for (int d = 1; d < 3; ++d) b.c[d] = a.c[d];
            b.c[0] = a.c[0] + std::max(std::max(a.w[0] + b.w[0], a.w[1] + b.w[1]), a.w[2] + b.w[2]) / angle;
        }
        a.sum = (a.w[0] + a.w[1]) + a.w[2];
        b.sum = (b.w[0] + b.w[1]) + b.w[2];
        for (int d = 0; d < 3; ++d) {
            fa.c[d] = (float)a.c[d]; fa.w[d] = (float)a.w[d];
            fb.c[d] = (float)b.c[d]; fb.w[d] = (float)b.w[d];
        }
        const bool an = q & 1, bn = (q & 2) || !an;
        const int r = walk_bound(fa, fb, an, bn, (float)(cutoff * cutoff), (float)(angle * angle));
        if (r == WALK_UNDECIDED) continue;
        ++decided;
        if (r != exact(a, b, an, bn, cutoff, angle)) ++wrong;
    }
    printf("%ld %ld %ld\n", wrong, decided, n);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("walk")
    (d / "w.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                           os.path.join(REPO, "photons-on-mt3000_b200", "csrc"), str(d / "w.cpp"), "-o", str(d / "w")])
    return str(d / "w")


@pytest.mark.parametrize("box", [1e-9, 1.0, 1e6, 1e20])
@pytest.mark.parametrize("angle", [0.0, 0.4, 1.5])
@pytest.mark.parametrize("offset", [0.0, 1.0, 1000.0])
def test_a_decided_pair_is_decided_as_in_fp64(program, box, angle, offset):
    wrong, decided, n = map(int, subprocess.check_output([program, str(box), str(angle), str(offset * box)],
                                                         text=True).split())
    assert wrong == 0
    if offset <= 1.0 and 1e-6 < box < 1e10:
        assert decided > 0.5 * n


# Boxes with one centre or width NaN or infinite: the exact test opens a pair whose
# gap is NaN (no comparison with NaN holds), so the bound may only leave it to that
# test; where it decides another pair, it decides the same.
NONFINITE = SOURCE.split("int main")[0] + r"""
#include <limits>
int main() {
    const double bad[] = {std::numeric_limits<double>::quiet_NaN(), std::numeric_limits<double>::infinity(),
                          -std::numeric_limits<double>::infinity()};
    long wrong = 0, n = 0;
    for (double value : bad)
        for (int at = 0; at < 12; ++at)            // which number of which box
            for (int gap = 0; gap < 8; ++gap)      // on which axes the boxes lie apart
                for (int kinds = 0; kinds < 4; ++kinds)
                    for (double angle : {0.0, 0.4}) {
                        WalkBox a, b;
                        WalkBox32 fa, fb;
                        for (int d = 0; d < 3; ++d) {
                            a.c[d] = 0.5;
                            b.c[d] = 0.5 + (gap >> d & 1 ? 5.0 : 0.0);
                            a.w[d] = b.w[d] = 0.25;
                        }
                        WalkBox &box = at < 6 ? a : b;
                        (at % 6 < 3 ? box.c : box.w)[at % 3] = value;
                        a.sum = (a.w[0] + a.w[1]) + a.w[2];
                        b.sum = (b.w[0] + b.w[1]) + b.w[2];
                        for (int d = 0; d < 3; ++d) {
                            fa.c[d] = (float)a.c[d]; fa.w[d] = (float)a.w[d];
                            fb.c[d] = (float)b.c[d]; fb.w[d] = (float)b.w[d];
                        }
                        const bool an = kinds & 1, bn = (kinds & 2) || !an;
                        const int r = walk_bound(fa, fb, an, bn, 0.01f, (float)(angle * angle));
                        if (r != WALK_UNDECIDED && (value != value || r != exact(a, b, an, bn, 0.1, angle))) ++wrong;
                        ++n;
                    }
    printf("%ld %ld\n", wrong, n);
}
"""


def test_a_box_that_is_not_finite_is_left_to_the_exact_test(tmp_path):
    (tmp_path / "n.cpp").write_text(NONFINITE)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                           os.path.join(REPO, "photons-on-mt3000_b200", "csrc"), str(tmp_path / "n.cpp"), "-o",
                           str(tmp_path / "n")])
    wrong, n = map(int, subprocess.check_output([str(tmp_path / "n")], text=True).split())
    assert n == 3 * 12 * 8 * 4 * 2 and wrong == 0
