"""Range of the tensor-core M2L's FP16 operators, on the CPU: the powers of two
of m2l_group.h, compiled here, bring every operator entry that the acceptance
test admits below FP16's largest number (65504), and are all 1 where no entry
comes near it.

An entry of output degree j and input degree n is, with d = j + n and the
offset v in units of the finer radius, at most c (d-m)! P_d^m(cos a) / |v|^(d+1)
(c = 2 for n > 0) times 2^(dl n) for a source dl levels coarser or
2^(dl (j + 1)) for one finer, and largest for m = d, where (d-m)! P_d^m is
(2d-1)!! sin^d a.  It is taken here at the integer offsets that exist (even
components between cells of one level, odd ones otherwise, the axis with the
smallest component vertical), not at the acceptance radius that the header
bounds it by."""
import itertools
import math
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "minimal_b200", "csrc")
PROGRAM = r"""
#include <cstdio>
#include "m2l_group.h"
int main(int argc, char **argv) {
  const fmm::TcScale s = fmm::make_tc_scale(atoi(argv[1]), atof(argv[2]), -4, 3, 1.7);
  printf("%d\n", (int)s.any);
  for (int n = 0; n < fmm::TC_MAX_P; n++) printf("%.17g %.17g\n", s.in[n], s.out[n]);
}
"""


@pytest.fixture(scope="module")
def scale(tmp_path_factory):
    d = tmp_path_factory.mktemp("tc_scale")
    (d / "s.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(d / "s.cpp"), "-o", str(d / "s")], check=True)

    def run(P, theta):
        v = subprocess.run([str(d / "s"), str(P), str(theta)], check=True, capture_output=True, text=True).stdout.split()
        return v[0] == "1", [float(x) for x in v[1::2]], [float(x) for x in v[2::2]]

    return run


def offsets(dl, theta):
    """The admissible offsets nearest to the acceptance radius, by gap."""
    lo = (1 + 2 ** abs(dl)) / theta
    parity = 1 if dl else 0
    for v in itertools.combinations_with_replacement(range(32), 3):  # ascending: v[0] vertical
        r = math.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
        if all(c % 2 == parity for c in v) and lo < r < 1.2 * lo + 2:
            yield math.hypot(v[1], v[2]), r


def largest(P, theta, s_in, s_out):
    worst = 0.0
    for dl in range(-4, 4):
        vs = list(offsets(dl, theta))
        for d in range(P if vs else 0):
            z = math.prod(range(1, 2 * d, 2)) * max(xy ** d / r ** (2 * d + 1) for xy, r in vs)
            for n in range(d + 1):
                j = d - n
                f = 2.0 ** (dl * n) if dl >= 0 else 2.0 ** (-dl * (j + 1))
                worst = max(worst, (2 if n else 1) * z * f / (s_in[n] * s_out[j]))
    return worst


@pytest.mark.parametrize("theta", [0.3, 0.4, 0.5, 0.6, 0.8, 1.0])
@pytest.mark.parametrize("P", [4, 8, 10, 11, 12, 13, 14, 15])
def test_operators_fit_fp16(scale, P, theta):
    some, s_in, s_out = scale(P, theta)
    plain = largest(P, theta, [1.0] * 16, [1.0] * 16)
    assert largest(P, theta, s_in, s_out) < 65504
    assert some or plain < 65504
    assert plain > 65504 / 8 or not some  # left alone well inside the range
    for f in s_in + s_out:
        assert f >= 1 and math.frexp(f)[0] == 0.5  # powers of two
    # the monopole keeps its scale, and the low degrees theirs where only
    # pairs of different levels need it
    assert s_in[0] == 1
    if theta <= 0.5 and P <= 13:
        assert max(s_in[:6] + s_out[:6]) == 1


def test_the_range_is_exceeded_without(scale):
    for P, theta in ((11, 0.5), (12, 0.4), (12, 0.5), (13, 0.4), (14, 0.5)):
        assert largest(P, theta, [1.0] * 16, [1.0] * 16) > 65504
    assert largest(10, 0.5, [1.0] * 16, [1.0] * 16) < 65504 and not scale(10, 0.5)[0]
