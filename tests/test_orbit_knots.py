"""The knot searches of csrc/orbit_knots.h, compiled for the host: both end for
every displacement (huge, infinite and NaN ones too), agree with each other
and with the knots counted in exact arithmetic, and fail from the same number
of knots on.  An endless search on the GPU would hang it, so this runs here."""
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from unstaggered_pic_b200 import build

CSRC = os.path.join(os.path.dirname(build.__file__), "csrc")
MAX_KNOTS = 38  # kMaxBreaks less the two ends

PROGRAM = r"""
#include <stdio.h>
#include "orbit_knots.h"
using namespace upic;
// per orbit: knots found by the list (-1: too many), by the walk, its segments, their total length
int main() {
    double ux, uy, dux, duy;
    while (scanf("%lf %lf %lf %lf", &ux, &uy, &dux, &duy) == 4) {
        double b[kMaxBreaks];
        int nb = 0;
        b[nb++] = 0.0;
        b[nb++] = 1.0;
        bool ok = fabs(dux) < 1.0e-300 || axis_breaks(ux, dux, b, nb);
        ok = ok && (fabs(duy) < 1.0e-300 || axis_breaks(uy, duy, b, nb));
        KnotWalk w;
        w.init(ux, uy, dux, duy);
        int knots = 0, segments = 0;
        double total = 0.0, sa, sb;
        for (;;) {
            if (w.nb > 0) knots = w.nb - 2;
            if (!w.next(ux, uy, dux, duy, sa, sb)) break;
            if (w.nb > 0) knots = w.nb - 2;
            ++segments;
            total += sb - sa;
        }
        printf("%d %d %d %.17g\n", ok ? nb - 2 : -1, w.nb == 0 ? knots : -1, segments, total);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def search(tmp_path_factory):
    d = tmp_path_factory.mktemp("knots")
    src, exe = d / "knots.cu", d / "knots"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc(), "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC, str(src), "-o", str(exe)],
                   check=True)

    def run(orbits):
        text = "\n".join(" ".join(float(v).hex() if math.isfinite(v) else str(v) for v in o) for o in orbits)
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True, timeout=20).stdout
        rows = [line.split() for line in out.splitlines()]
        return [(int(a), int(b), int(c), float(t)) for a, b, c, t in rows]

    return run


def knots_between(u, du):
    """Integers strictly between u and u + du."""
    a, b = sorted((Fraction(u), Fraction(u) + Fraction(du)))
    return max(0, math.ceil(b) - math.floor(a) - 1)


@pytest.mark.parametrize("du", [1e13, 1e24, 1e30, 1e300, math.inf])
@pytest.mark.parametrize("sign", [1, -1])
def test_huge_displacements_fail_at_once(search, du, sign):
    got = search([(3.25, 5.5, sign * du, 0.1), (3.25, 5.5, 0.1, sign * du), (3.0, 0.0, sign * du, sign * du)])
    for listed, walked, segments, _ in got:
        assert (listed, walked, segments) == (-1, -1, 0)


def test_nan_displacements_end(search):
    # no knot is found in them: one segment over the whole orbit, whose values are NaN
    for listed, walked, segments, total in search([(3.25, 5.5, math.nan, 0.1), (3.25, 5.5, 0.1, math.nan)]):
        assert (listed, walked, segments, total) == (0, 0, 1, 1.0)


def test_knots_of_ordinary_orbits(search):
    """Counts up to and past the limit, from both sides of the early refusal (64
    cells) and from points on a knot."""
    rng = np.random.default_rng(7)
    orbits = [(u, w, du, dw) for u, w, du, dw in zip(rng.uniform(0, 64, 400), rng.uniform(0, 64, 400),
                                                     rng.uniform(-45, 45, 400), rng.uniform(-3, 3, 400))]
    orbits += [(0.5, 0.5, s * d, 0.0) for d in (0.25, 1.0, 37.75, 38.75, 39.25, 63.75, 64.25, 65.0) for s in (1, -1)]
    orbits += [(4.0, 7.0, s * 2.5, t * 0.5) for s in (1, -1) for t in (1, -1)]
    orbits += [(0.25, 0.75, 1e-17, -1e-17), (0.25, 0.75, 0.0, 0.0)]
    for o, (listed, walked, segments, total) in zip(orbits, search(orbits)):
        n = knots_between(o[0], o[2]) + knots_between(o[1], o[3])
        want = n if n <= MAX_KNOTS else -1
        assert (listed, walked) == (want, want), o
        if want >= 0:
            assert segments == want + 1 and abs(total - 1.0) < 1e-12, o
