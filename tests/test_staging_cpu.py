"""The buffers entry points keep between calls, on the host (no GPU): after an allocation that failed, a
smaller call must not take the old capacity for a buffer that is gone."""
import os
import subprocess

import pytest

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "fastcorticalwiring_b200", "csrc")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("staging") / "staging_check")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", CSRC, "-o", exe,
                           os.path.join(ROOT, "tests", "staging_check.cpp")])
    return exe


@pytest.mark.parametrize("limit,needs,want", [
    (100, (10, 5, 20, 20), ["0:10", "0:10", "0:20", "0:20"]),
    (100, (50, 200, 40, 200, 10), ["0:50", "7:0", "0:40", "7:0", "0:10"]),  # out of memory, then smaller calls
    (100, (200, 1), ["7:0", "0:1"]),
])
def test_capacity_follows_the_buffer(checker, limit, needs, want):
    out = subprocess.check_output([checker, str(limit), *map(str, needs)], text=True)
    assert out.split() == want
