"""The device-wide scan on the host, its kernels' source compiled with the CUDA built-ins emulated: sizes about
the tile (4096 counts) and the one-CTA limit (8192), and CTAs whose wait for the others runs out."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "brig-join_b200", "csrc")


@pytest.fixture(scope="module")
def scan(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("scan") / "scan")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-o", exe, os.path.join(HERE, "scan_host.cpp")], check=True)
    return lambda *a: subprocess.run([exe, *map(str, a)], check=True, capture_output=True, text=True).stdout.strip()


@pytest.mark.parametrize("n", [1, 511, 4095, 4096, 4097, 8191, 8192])
def test_one_cta(scan, n):
    assert scan(n, 1, 0, 0) == "ok"


@pytest.mark.parametrize("n,grid", [(8193, 3), (12_288, 3), (12_289, 4), (50_001, 5), (200_000, 49)])
@pytest.mark.parametrize("polls,reverse", [(0, 0), (100, 0), (100, 1)])
def test_many_ctas(scan, n, grid, polls, reverse):
    """CTAs that find the sums before theirs, and CTAs whose wait for them runs out: these add up what lies
    before their share themselves."""
    assert scan(n, grid, polls, reverse) == "ok"
