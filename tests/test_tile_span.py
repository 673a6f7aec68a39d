"""The column intervals of the screen-block lists (tile_span.h), compiled for
the CPU, against the tile test they stand in for: no tile decided wrongly over
round, long, axis-aligned and diagonal splats, all tile shapes and odd
viewports, and few tiles left to the test."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("span") / "tile_span_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "cindergs_b200", "csrc"),
                    os.path.join(ROOT, "tests", "tile_span_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_spans_agree_with_the_tile_test(check, seed):
    out = subprocess.run([check, "1500000", str(seed)], check=True, capture_output=True, text=True)
    wrong, left_open, rows, tests = (int(x) for x in out.stdout.split())
    assert tests > 1_000_000
    assert wrong == 0
    assert left_open < 0.01 * rows
