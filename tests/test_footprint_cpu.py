"""A proof's scratch stays within what its key reserves (bg_prove_footprint), whatever the header: host
logic of the library, no GPU."""
import os
import random
import shutil
import subprocess

import pytest

from conftest import PKG

SRC = r"""
#include "prove.h"
#include <cstdio>
using namespace bg;
int main() {
  Header h;
  while (scanf("%u %u %u %u %u %u", &h.nc, &h.ni, &h.nw, &h.lg, &h.nh, &h.nl) == 6) {
    h.na = h.nb = h.ni + h.nw;
    const int c[5] = {msm_pick_c_table(h.na, false), msm_pick_c_table(h.nb, false), msm_pick_c_table(h.nb, true),
                      msm_pick_c_table(h.nh, false), msm_pick_c_table(h.nl, false)};
    const int cap = prove_round_cap(h, c);
    printf("%zu %zu %zu %d %zu\n", prove_footprint(h), prove_scratch(h, c, 0), prove_scratch(h, c, 2), cap,
           prove_scratch(h, c, cap));
  }
}
"""


@pytest.fixture(scope="module")
def sizes(built_lib, tmp_path_factory):
    """headers (nc, ni, nw, lg, nh, nl) -> footprint, scratch without rounds, with two, cap, with cap"""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    d = tmp_path_factory.mktemp("footprint")
    (d / "t.cpp").write_text(SRC)
    exe = str(d / "t")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", inc, "-I", os.path.join(PKG, "csrc"), "-o", exe, str(d / "t.cpp"),
                    "-L", PKG, "-lbg", "-Wl,-rpath," + PKG, "-Wl,--allow-shlib-undefined"], check=True)

    def run(headers):
        text = "\n".join(" ".join(map(str, h)) for h in headers)
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return run


def square_chain(k):
    n = 1 << k
    return (n, 2, n, k + 1, 2 * n - 1, n)


def test_scratch_of_any_header_stays_within_the_reservation(sizes):
    rng = random.Random(80)
    headers = []
    for _ in range(4000):
        nz, lg = int(2 ** rng.uniform(1, 21.5)) + 1, rng.randint(0, 21)
        d = 1 << lg
        ni = rng.randint(1, min(nz, d))
        nw = nz - ni
        headers.append((rng.randint(0, d - ni), ni, nw, lg, rng.choice([d - 1, d, d // 2, 0, rng.randint(0, d)]),
                        rng.choice([nw, nw // 2, 0, rng.randint(0, nw)])))
    got = sizes(headers)
    assert len(got) == len(headers)
    for h, (reserved, none, two, cap, used) in zip(headers, got):
        assert used <= reserved, h
        assert none <= 0.8 * reserved, h  # what proofs took before their tables had pair rounds
    assert any(two > reserved for reserved, _, two, _, _ in got)  # the rule is needed
    assert {cap for _, _, two, cap, _ in got} == {0, 1, 2}


def test_square_chains_keep_their_rounds(sizes):
    for k, (reserved, _, two, cap, _) in zip(range(8, 21), sizes([square_chain(k) for k in range(8, 21)])):
        assert cap == 2 and two <= reserved, k


@pytest.mark.parametrize("k,reserved", [(10, 29617609), (14, 267818456), (18, 1469374112), (20, 7746652583)])
def test_a_budget_admits_what_it_admitted(sizes, k, reserved):
    """the reservation does not move when widths or rounds are tuned"""
    assert sizes([square_chain(k)])[0][0] == reserved
