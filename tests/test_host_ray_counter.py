"""The counter from which traversal lanes take rays (host/ray_counter.h), run on the CPU
with every lane of a GPU taking once more after the last ray: each ray is taken once and
no index lies outside them, up to the largest number of rays that a call takes."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r'''
#include "ray_counter.h"
#include <climits>
#include <cstdio>
#include <cstdlib>
int main(int, char **argv) {
    const int n = std::atoi(argv[1]);
    const int lanes = 148 * 2048;
    int counter = n > 100 ? n - 100 : 0;  // where the last rays are handed out
    const unsigned first = unsigned(counter);
    long taken = 0, wrong = 0;
    for (int group = 0; group < lanes / 32 + 4; group++) {
        for (int rank = 0; rank < 32; rank++) {
            const unsigned k = lambda_host::taken_index(counter, rank);
            if (!lambda_host::item_left(k, n)) continue;
            taken++;
            wrong += k < first || k >= unsigned(n) || int(k) < 0;
        }
        counter = int(unsigned(counter) + 32u);  // what atomicAdd leaves
    }
    std::printf("%ld %ld\n", taken, wrong);
}
'''


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("counter")
    (d / "counter.cpp").write_text(PROGRAM)
    inc = os.path.join(ROOT, "lambda_b200", "csrc", "host")
    subprocess.run(["g++", "-std=c++20", "-O1", "-I", inc, str(d / "counter.cpp"), "-o", str(d / "counter")], check=True)
    return str(d / "counter")


@pytest.mark.parametrize("n", [1, 31, 32, 1000, 2**31 - 300_000, 2**31 - 128, 2**31 - 33, 2**31 - 1])
def test_each_ray_is_taken_once(program, n):
    out = subprocess.run([program, str(n)], capture_output=True, text=True, check=True).stdout.split()
    assert out == [str(min(n, 100)), "0"]
