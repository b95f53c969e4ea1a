"""CPU: the rule that picks an automatic grid's step (csrc/wf_price.h, compiled
here on its own) against times measured on a B200 in every form, microseconds a
step: grids whose x extent leaves bricks or tiles partly outside, thin and deep
slabs on some axes or all, periodic axes, both storage widths.

The tolerance is the spread of those times: a form repeated in the same process
differs by up to 7 % (memory that another grid used before), so a pick within
8 % of the best counts as right."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wavefront_b200", "csrc")
FORMS = ("split", "march", "brick", "mix")

# nx, ny, nz, CPML depths, periodic axes, 16-bit, {form: us}
MEASURED = [
    (16, 256, 256, (0, 0, 0), '', False, {"split": 23.0, "march": 62.7, "brick": 27.1}),
    (16, 256, 256, (0, 0, 0), 'x', False, {"split": 22.8, "brick": 37.6}),
    (16, 256, 256, (0, 0, 0), 'xy', False, {"split": 22.8, "brick": 37.8}),
    (16, 256, 256, (0, 0, 0), 'xyz', False, {"split": 22.8, "brick": 38.1}),
    (24, 256, 256, (0, 0, 0), 'x', False, {"split": 32.1, "brick": 36.8}),
    (24, 256, 256, (0, 0, 0), 'yz', False, {"split": 31.5, "brick": 26.7}),
    (256, 256, 256, (0, 0, 0), 'xyz', False, {"split": 384.0, "brick": 206.9}),
    (192, 160, 256, (0, 0, 0), 'xy', False, {"split": 185.4, "brick": 97.1}),
    (104, 104, 104, (0, 0, 0), 'yz', False, {"split": 23.4, "brick": 18.0}),
    (560, 8, 8, (0, 0, 0), 'yz', False, {"split": 6.7, "brick": 5.0}),
    (40, 128, 128, (4, 4, 4), '', False, {"split": 22.6, "march": 56.0, "brick": 19.4}),
    (40, 200, 264, (0, 0, 0), '', False, {"split": 43.3, "march": 55.5, "brick": 35.6}),
    (72, 320, 256, (10, 10, 10), '', False, {"split": 176.9, "march": 251.1, "brick": 157.3}),
    (104, 440, 320, (0, 0, 0), '', False, {"split": 338.1, "march": 148.1, "brick": 184.7}),
    (136, 440, 320, (10, 10, 10), '', False, {"split": 520.7, "march": 454.1, "brick": 384.3, "mix": 432.2}),
    (136, 128, 128, (0, 0, 0), '', False, {"split": 46.7, "march": 39.0, "brick": 29.8}),
    (160, 160, 160, (0, 0, 0), '', False, {"split": 101.1, "march": 56.5, "brick": 45.7}),
    (264, 440, 320, (10, 10, 10), '', False, {"split": 968.5, "march": 595.8, "brick": 637.8, "mix": 620.2}),
    (264, 440, 320, (24, 24, 24), '', False, {"split": 1019.4, "march": 812.9, "brick": 633.0, "mix": 640.0}),
    (328, 440, 320, (10, 10, 10), '', False, {"split": 1183.8, "march": 709.1, "brick": 755.0, "mix": 682.6}),
    (328, 440, 320, (32, 32, 32), '', False, {"split": 1288.2, "march": 926.5, "brick": 773.2, "mix": 788.9}),
    (64, 64, 64, (16, 16, 16), '', False, {"split": 13.6, "march": 51.0, "brick": 6.5}),
    (256, 256, 256, (8, 8, 8), '', False, {"split": 446.8, "march": 297.2, "brick": 235.1, "mix": 235.4}),
    (384, 384, 384, (0, 0, 0), '', False, {"split": 1266.6, "march": 452.5, "brick": 627.4}),
    (512, 512, 512, (8, 8, 8), '', False, {"split": 3387.1, "march": 1380.7, "brick": 1764.8, "mix": 1417.0}),
    (512, 512, 512, (16, 16, 16), '', False, {"split": 3455.2, "march": 1620.7, "brick": 1832.6, "mix": 1527.9}),
    (512, 512, 512, (0, 0, 16), '', False, {"split": 3097.4, "march": 1115.7, "brick": 1729.3}),
    (640, 640, 640, (10, 10, 10), '', False, {"split": 6539.0, "march": 2618.5, "brick": 3700.8, "mix": 2885.8}),
    (1024, 1024, 1024, (8, 8, 8), '', False, {"split": 26250.2, "march": 10214.1, "brick": 13943.6, "mix": 10589.5}),
    (128, 128, 128, (48, 48, 48), '', False, {"split": 94.9, "brick": 54.3}),
    (256, 256, 256, (36, 36, 36), '', False, {"split": 523.0, "brick": 295.8}),
    (256, 256, 256, (0, 0, 0), '', True, {"march": 123.9, "brick": 143.8}),
    (384, 264, 304, (0, 0, 0), '', True, {"march": 223.8, "brick": 266.4}),
    (360, 200, 264, (0, 0, 0), '', True, {"march": 160.4, "brick": 178.8}),
    (320, 320, 320, (16, 16, 16), '', True, {"march": 624.8, "brick": 462.6, "mix": 387.7}),
    (64, 64, 64, (10, 10, 10), '', True, {"march": 149.2, "brick": 12.4}),
    (512, 512, 512, (16, 16, 16), '', True, {"march": 1497.3, "brick": 1745.9, "mix": 1391.0}),
    (200, 200, 200, (4, 4, 4), '', True, {"march": 243.7, "brick": 133.1, "mix": 133.8}),
    (392, 512, 288, (7, 0, 0), '', False, {"march": 576.6, "brick": 854.7, "mix": 670.3}),
]

MAIN = r'''
#include "wf_price.h"
#include <cstdio>
int main() {
  int n[3], t[3], p[3], b, march;
  while (scanf("%d%d%d%d%d%d%d%d%d%d%d", n, n + 1, n + 2, t, t + 1, t + 2, p, p + 1, p + 2, &b, &march) == 11) {
    wf::StepShape s{{n[0], n[1], n[2]}, {t[0], t[1], t[2]}, {p[0] != 0, p[1] != 0, p[2] != 0}, b != 0};
    printf("%d\n", static_cast<int>(wf::cheapest_step(s, march != 0, true, true)));
  }
}
'''


@pytest.fixture(scope="module")
def pick(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("price")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", CSRC, str(d / "main.cpp"), "-o", str(d / "pick")], check=True)

    def run(cases):
        lines = "".join(" ".join(str(int(v)) for v in c) + "\n" for c in cases)
        out = subprocess.run([str(d / "pick")], input=lines, capture_output=True, text=True, check=True).stdout
        return [FORMS[int(v)] for v in out.split()]

    return run


def test_the_pick_is_the_fastest_measured_form(pick):
    cases = []
    for nx, ny, nz, depth, per, b16, us in MEASURED:
        march = not per and all(min(2 * t, n) <= 64 for t, n in zip(depth, (nx, ny, nz)))
        cases.append((nx, ny, nz, *depth, *(a in per for a in "xyz"), b16, march))
    bad = []
    for c, m, form in zip(cases, MEASURED, pick(cases)):
        us = m[-1]
        if us[form] > 1.08 * min(us.values()):
            bad.append((m[:-1], form, us))
    assert not bad, bad


def test_marching_and_bricks_stay_within_what_can_run(pick):
    # nothing marches on periodic axes or over slabs of more than 64 positions
    got = pick([(512, 512, 512, 0, 0, 0, 0, 1, 1, 0, 0), (256, 256, 256, 40, 40, 40, 0, 0, 0, 0, 0)])
    assert all(f in ("split", "brick") for f in got)


# (grids, cells of an edge, CPML depth, us as bricks, us as marching items)
BATCHES = [
    (4, 256, 0, 932.3, 576.9), (4, 256, 10, 1115.3, 1379.9), (4, 256, 8, 1017.0, 939.5), (3, 320, 16, 1534.5, 1629.4),
    (16, 128, 0, 460.2, 302.3), (16, 128, 10, 641.1, 974.1), (20, 104, 0, 381.5, 223.8), (48, 40, 0, 85.8, 91.8),
    (48, 40, 4, 115.0, 215.8), (32, 72, 0, 225.3, 163.9), (32, 72, 8, 296.0, 401.6), (3, 64, 10, 24.6, 100.3),
    (3, 32, 0, 6.8, 25.2), (60, 96, 0, 734.4, 527.6), (60, 96, 8, 961.2, 1194.2), (1, 512, 8, 1927.8, 1568.5),
    (1, 448, 0, 1252.9, 844.2), (60, 24, 4, 37.7, 132.2),
]

BATCH_MAIN = r'''
#include "wf_price.h"
#include <cstdio>
#include <vector>
int main() {
  int n, e, t;
  while (scanf("%d%d%d", &n, &e, &t) == 3) {
    const std::vector<wf::StepShape> v(n, wf::StepShape{{e, e, e}, {t, t, t}, {}, false});
    printf("%d\n", wf::batch_takes_bricks(v.data(), n) ? 1 : 0);
  }
}
'''


def test_a_batch_takes_the_faster_measured_form(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    (tmp_path / "batch.cpp").write_text(BATCH_MAIN)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", CSRC, str(tmp_path / "batch.cpp"), "-o", str(tmp_path / "batch")],
                   check=True)
    lines = "".join(f"{n} {e} {t}\n" for n, e, t, _, _ in BATCHES)
    out = subprocess.run([str(tmp_path / "batch")], input=lines, capture_output=True, text=True, check=True).stdout
    for (n, e, t, bricks, march), v in zip(BATCHES, out.split()):
        assert (bricks if v == "1" else march) <= 1.08 * min(bricks, march), (n, e, t, v)
