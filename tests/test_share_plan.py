"""csrc/share_plan.cuh: on how many CTAs a decode product runs.  No GPU needed."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gllm-kernels_b200", "csrc")


@pytest.fixture(scope="module")
def decode_ctas(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("plan")
    (d / "t.cpp").write_text('#include "share_plan.cuh"\n#include <cstdio>\n#include <cstdlib>\n'
                             'int main(int c, char **v) { for (int i = 1; i + 5 < c; i += 6) std::printf("%lld\\n", (long long)gllmk::decode_ctas('
                             'std::atoll(v[i]), std::atoll(v[i + 1]), std::atoi(v[i + 2]), std::atoll(v[i + 3]), std::atoi(v[i + 4]) != 0, std::atoi(v[i + 5]) != 0)); }\n')
    exe = d / "t"
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-x", "c++", str(d / "t.cpp"), "-o", str(exe)], check=True)

    def call(cases):
        args = [str(int(a)) for c in cases for a in c]
        return [int(l) for l in subprocess.run([str(exe), *args], capture_output=True, text=True, check=True).stdout.split()]
    return call


def test_three_units_in_few_ctas_stay_on_the_resident_grid(decode_ctas):
    """Measured 1 to 34 % slower on 318 CTAs of three units than on 444 of two or three (rows of 4 to 56 blocks)."""
    cases = [(952, 444, 3, nb, several, tiled) for nb in (4, 8, 12, 14, 16, 20, 28, 32, 43, 56) for several in (0, 1) for tiled in (0, 1)]
    assert decode_ctas(cases) == [444] * len(cases)


def test_four_units_whose_shares_do_not_end_with_the_row_stay_on_the_resident_grid(decode_ctas):
    cases = [(1400, 444, 3, nb, several, tiled) for nb in (12, 14, 24, 43) for several in (0, 1) for tiled in (0, 1)] + [(1400, 444, 3, 16, 1, 1)]
    assert decode_ctas(cases) == [444] * len(cases)


def test_where_the_smaller_grid_is_the_faster_one(decode_ctas):
    cases = [(1376, 444, 3, 16, 0, 1), (1376, 444, 3, 16, 1, 0), (1400, 444, 3, 4, 1, 1), (952, 296, 2, 14, 0, 1), (704, 296, 2, 32, 0, 1), (512, 444, 3, 16, 1, 1)]
    assert decode_ctas(cases) == [344, 344, 350, 238, 235, 256]
    # two units: not with one column group, not on short rows, not when only a few CTAs have two
    assert decode_ctas([(512, 444, 3, 16, 0, 1), (512, 444, 3, 8, 1, 1), (448, 444, 3, 16, 1, 0)]) == [444] * 3


def test_every_share_is_at_most_the_longest_and_no_cta_is_idle(decode_ctas):
    cases = [(u, c, s, nb, v, t) for u in (1, 2, 147, 148, 149, 443, 444, 445, 888, 889, 1332, 1333, 1776, 1777, 5000, 10 ** 7)
             for c, s in ((148, 1), (296, 2), (444, 3)) for nb in (1, 4, 12, 16, 43, 112) for v in (0, 1) for t in (0, 1)]
    for (u, c, s, nb, v, t), got in zip(cases, decode_ctas(cases)):
        assert 1 <= got <= min(u, c)
        assert -(-u // got) == -(-u // min(u, c))  # the longest share is what it was
