"""Which bases without a group get two-table ranks (csrc/ranks.h, compiled by the host compiler): the
table words are 32 bits wide, so a basis of more than 2^32 states keeps the search."""

import math
import os
import shutil
import subprocess

import pytest

from conftest import REPO

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "ranks.h"
int main(int argc, char** argv) {
  lsg::RankTables t;
  const bool ok = lsg::rank_tables_for(atoi(argv[1]), atoi(argv[2]), atoi(argv[3]), atoi(argv[4]) != 0, &t);
  printf("%d %lld %d %d\n", (int)ok, (long long)t.states, t.split, t.high_bits);
}
"""


@pytest.fixture(scope="module")
def tables(tmp_path_factory):
    compiler = shutil.which("g++") or shutil.which("c++")
    if compiler is None:
        pytest.skip("no host compiler")
    folder = tmp_path_factory.mktemp("ranks")
    source, program = folder / "ranks.cpp", folder / "ranks"
    source.write_text(PROGRAM)
    subprocess.run([compiler, "-std=c++17", "-I", os.path.join(REPO, "lattice-symmetries_gb300", "csrc"), str(source),
                    "-o", str(program)], check=True)

    def run(bits, weight, up=-1, inversion=False):
        out = subprocess.run([str(program), str(bits), str(weight), str(up), str(int(inversion))], check=True,
                             capture_output=True, text=True).stdout.split()
        return bool(int(out[0])), int(out[1]), int(out[2]), int(out[3])

    return run


@pytest.mark.parametrize("bits,weight,inversion,expected", [
    (34, 17, False, True),   # 2.33e9 states
    (35, 17, False, False),  # 4.54e9: more than 2^32
    (36, 18, False, False),
    (36, 18, True, False),   # 4.54e9
    (34, 17, True, True),
    (40, 3, False, True),
    (40, 20, False, False),
    (41, 2, False, False),   # tables of more than 2^20 words
    (7, 0, False, True),
    (7, 7, False, True),
])
def test_fixed_weight(tables, bits, weight, inversion, expected):
    ok, states, split, high = tables(bits, weight, -1, inversion)
    assert ok == expected
    if bits <= 40:
        assert states == math.comb(bits, weight) // (2 if inversion else 1)
        assert split + high == bits


@pytest.mark.parametrize("sites,up,down,expected", [(18, 9, 9, True), (20, 10, 10, False), (20, 5, 8, True),
                                                    (20, 0, 20, True)])
def test_two_species(tables, sites, up, down, expected):
    ok, states, split, high = tables(2 * sites, up + down, up)
    assert ok == expected and split == high == sites
    assert states == math.comb(sites, up) * math.comb(sites, down)
    assert (states <= 2 ** 32) == expected
