"""The bounds of the version-5 sweep's waits (csrc/lu5_wait.h), on the host: warp E's rounds follow the
handle's limit, the tries of the other roles outlast them for every limit, and both are finite."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "opencfd-ec_b200", "csrc")
PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "lu5_wait.h"
int main(int argc, char** argv) {
  for (int q = 1; q < argc; q++) std::printf("%d %d\\n", ocfd::lu5_rounds(std::atoll(argv[q])), ocfd::lu5_tries(std::atoll(argv[q])));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("lu5_wait")
    src = d / "wait.cpp"
    src.write_text(PROGRAM)
    subprocess.check_call([os.environ.get("CXX", "g++"), "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(d / "wait")])
    return str(d / "wait")


def test_the_other_roles_outlast_the_wait_between_tiles(program):
    limits = [0, 1, 7, 8, 4000, 4000000, 2 ** 31, 2 ** 40, 2 ** 63 - 1]
    out = subprocess.run([program] + [str(v) for v in limits], capture_output=True, text=True, check=True).stdout.split()
    for limit, rounds, tries in zip(limits, map(int, out[::2]), map(int, out[1::2])):
        assert rounds == min(limit // 8, 2 ** 30)
        assert rounds + 25000 == tries < 2 ** 31   # a try in vain (3.95 us) takes longer than a round
