"""The rules by which CTAs exchange data without a barrier around every access (csrc/sync_rules.h,
the functions the kernels use), run through random orders of events on the CPU."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("sync") / "check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "seemps2_gb300", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "sync_rules_check.cpp")], check=True)
    return lambda mode: subprocess.run([exe, mode], check=True, capture_output=True, text=True).stdout.strip()


def test_jacobi_block_rounds(check):
    """Clusters of 2 to 16 CTAs, three sweeps: every pair of blocks meets once a sweep, no block is
    written over while a copy of it may be in flight or its CTA works on it, and every wait ends,
    with reports of receipt or with buffers apart for what is sent. Without either, the check finds
    the write over a copy's source."""
    assert check("jacobi") == "ok"
    assert check("jacobi-outs") == "ok"
    assert check("jacobi-blind").endswith("a write over the source of a copy in flight")


@pytest.mark.parametrize("kernel", ["qr-step", "qr-batch"])
def test_householder_grid_sums(check, kernel):
    """1 to 64 steps: no sum is written over while a slower CTA may still read it.  With one buffer
    the check finds it: at any step, or where the last batch is a single step (5, 9, .. steps)."""
    assert check(kernel) == "ok"
    assert check(kernel + "-single").endswith("a sum written over while it is read")
