"""Plane ranges of single-patch launches (csrc/dn_range.h): the model's choice
against stage times measured on a B200."""
import os
import shutil
import subprocess

import pytest

from drnum_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))

# precision, cells, range of the fixed rule before (about four waves of at least
# eight planes), us a stage by range; periodic patches
MEASURED = [
    (64, (97, 61, 83), 8, {1: 139.8, 2: 121.4, 4: 114.5, 8: 109.3, 12: 134.3, 17: 160.6}),
    (64, (61, 101, 47), 8, {1: 100.4, 2: 88.0, 3: 86.4, 4: 99.0, 6: 86.0, 8: 92.7, 16: 148.3}),
    (64, (64, 64, 64), 8, {1: 68.1, 2: 59.9, 3: 69.6, 4: 61.0, 8: 81.1, 16: 132.3}),
    (64, (96, 96, 96), 8, {2: 186.4, 4: 173.8, 6: 169.1, 8: 188.6, 12: 163.8, 16: 183.4}),
    (64, (128, 128, 128), 10, {4: 388.2, 7: 375.3, 8: 385.9, 10: 377.8, 14: 368.9, 15: 371.4, 19: 427.1, 28: 404.0}),
    (64, (16, 65, 34), 8, {1: 23.2, 2: 27.1, 4: 39.2, 8: 69.4}),
    (32, (45, 198, 167), 8, {1: 136.1, 2: 108.6, 6: 89.6, 8: 94.5, 15: 98.8}),
    (32, (159, 157, 220), 10, {8: 246.3, 10: 242.5, 12: 241.8, 13: 240.1, 20: 243.2, 40: 249.9}),
    (32, (32, 32, 32), 8, {1: 10.7, 2: 14.7, 4: 20.9, 8: 35.3, 16: 64.9}),
    (32, (64, 64, 64), 8, {1: 25.0, 2: 18.9, 4: 20.9, 8: 33.2, 16: 59.8}),
    (32, (125, 67, 93), 8, {1: 80.4, 4: 62.3, 7: 57.3, 8: 63.3, 16: 78.3}),
    (32, (146, 67, 59), 8, {2: 55.6, 3: 53.8, 5: 48.0, 6: 52.9, 8: 63.3, 16: 78.0}),
    (32, (160, 160, 160), 8, {6: 171.2, 8: 162.4, 14: 149.7, 16: 167.3, 32: 160.1}),
    (32, (40, 200, 200), 8, {6: 89.5, 8: 97.5, 12: 81.5, 14: 88.9, 16: 100.3, 40: 179.4}),
    (32, (256, 256, 256), 26, {16: 558.4, 26: 552.5, 29: 539.0, 32: 541.8, 64: 598.5}),
]


@pytest.fixture(scope="module")
def chosen(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("ranges") / "plane_ranges")
    subprocess.run([shutil.which("g++"), "-O2", "-std=c++17", "-I", build.CSRC, "-o", exe,
                    os.path.join(HERE, "plane_ranges.cpp")], check=True)

    def run(patches):
        text = "\n".join("%d %d %d %d" % (p, *n) for p, n in patches)
        res = subprocess.run([exe], input=text, capture_output=True, text=True, check=True)
        return [[int(x) for x in line.split()] for line in res.stdout.splitlines()]
    return run


def test_choice_against_measured_times(chosen):
    """Within 10 % of the fastest measured range and 1 % (two runs of one side
    differ by up to 0.6 %) of the fixed rule's."""
    for (prec, n, old, us), (ic, *_) in zip(MEASURED, chosen([(p, n) for p, n, _, _ in MEASURED])):
        assert ic in us, (prec, n, ic)
        assert us[ic] <= 1.10 * min(us.values()) and us[ic] <= 1.01 * us[old], (prec, n, ic, us)


def test_range_bounds(chosen):
    """Every patch gets ranges of at least a plane that its extent and the
    grid's third extent (65535) allow."""
    patches = [(p, n) for p in (32, 64) for n in [(1, 1, 1), (1, 500, 3), (2, 1, 1), (7, 3, 100000), (100000, 1, 1),
                                                  (300000, 5, 2), (65535, 1, 1), (65536, 4, 32), (40, 2000, 2000)]]
    for (p, n), ranges in zip(patches, chosen(patches)):
        assert 2 <= len(ranges) <= 7 and len(set(ranges[1:])) == len(ranges) - 1, (p, n, ranges)
        for ic in ranges:
            assert 1 <= ic <= n[0] and -(-n[0] // ic) <= 65535, (p, n, ranges)
