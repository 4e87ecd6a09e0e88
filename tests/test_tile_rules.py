"""How products are cut for the device's SMs (csrc/tile_rules.h), on the CPU."""

import math
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "tile_rules.h"
int main(int, char** v) {
  int a[6];
  while (std::scanf("%d %d %d %d %d %d", a, a + 1, a + 2, a + 3, a + 4, a + 5) == 6) {
    const sm::GemmCut c = sm::gemm_cut(a[0], a[1], a[2], a[3], a[4]);
    std::printf("%d %d %d\n", c.tile, c.slices, sm::sgemm_slices((long)a[0] * a[1], a[2], 32, a[4]));
  }
}
"""


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    d = tmp_path_factory.mktemp("tiles")
    (d / "main.cpp").write_text(MAIN)
    exe = str(d / "main")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "seemps2_gb300", "csrc"), "-o", exe,
                    str(d / "main.cpp")], check=True)

    def run(cases):
        text = "\n".join(" ".join(map(str, c)) + " 0" for c in cases)
        out = subprocess.run([exe], input=text, check=True, capture_output=True, text=True).stdout
        return [tuple(map(int, l.split())) for l in out.splitlines()]

    return run


@pytest.mark.parametrize("sms", [1, 20, 76, 148, 152])
def test_least_work_for_the_fullest_sm(cut, sms):
    sizes = [(1, 1, 1), (16, 16, 16), (32, 33, 31), (130, 130, 256), (174, 174, 190), (300, 7, 2000), (600, 600, 40)]
    cases = [(*s, c, sms) for s in sizes for c in (0, 1)]
    for (M, N, K, cplx, _), (tile, slices, nz) in zip(cases, cut(cases)):
        def cost(t, z):
            kc = -(-(-(-K // z)) // 16) * 16
            one = 0.5 * t * t * kc * (4 if cplx else 1) + 1500
            return math.ceil(-(-M // t) * -(-N // t) * z / sms) * one + (1500 if z > 1 else 0)
        plans = [(t, z) for t in (16, 32) for z in range(1, 9) if z == 1 or K > 16 * (z - 1)]
        assert (tile, slices) in plans
        assert cost(tile, slices) == min(cost(*p) for p in plans)
        # predictor products of M x N tiles: two CTAs to an SM, slices of 32 and more
        assert nz in (1, 2, 4, 8) and (nz == 1 or K > 32 * nz // 2)
        assert nz == 8 or M * N * nz >= 2 * sms or K <= 32 * nz
        assert nz == 1 or M * N * nz // 2 < 2 * sms


def test_the_sm_count_decides(cut):
    """130 x 130 x 256: 150 CTAs on 152 SMs; on half as many SMs another cut."""
    a, b = cut([(130, 130, 256, 0, 152), (130, 130, 256, 0, 76)])
    assert a[:2] == (32, 6) and b[:2] != a[:2]
