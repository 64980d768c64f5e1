"""The short cosine of a bounded argument equals the general one bit for bit:
the source of both, compiled for the host, over whole binades around the
quarter turns, around large integers and half integers, and over every 257th
binary32 below the limit of 2^126, of both signs."""
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent
HEADER = ROOT.parent / "parallelparticleswarms.jl_gb300" / "csrc" / "pps_device.cuh"


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("cos")
    text = HEADER.read_text()
    odd = re.search(r"__device__ __forceinline__ bool is_odd_integer\(.*?\n}\n", text, re.S).group(0)
    a = text.index("constexpr float kCosP0")
    b = text.index("__device__ __forceinline__ float sin2pi(")
    (d / "cosines.inc").write_text(odd + text[a:b])
    exe = d / "check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(d), "-o", str(exe),
                    str(ROOT / "host" / "cos2pi_box_check.cpp")], check=True)

    def run(first, last, step):
        out = subprocess.run([str(exe), hex(first), hex(last), str(step)], check=True, capture_output=True, text=True)
        count, bad = map(int, out.stdout.split())
        assert count > 0 and bad == 0, (hex(first), count, bad)
    return run


@pytest.mark.parametrize("binade", [0x3E000000, 0x3E800000, 0x3F000000, 0x3F800000])  # 1/8, 1/4, 1/2, 1
def test_whole_binades(check, binade):
    check(binade, binade + 0x800000, 1)


def test_around_the_last_fractions(check):
    for exponent in range(0x40000000, 0x4C000000, 0x800000):
        check(exponent, exponent + 65536, 1)
        check(exponent + 0x7F0000, exponent + 0x800000, 1)


def test_every_magnitude_below_the_limit(check):
    check(0, 0x7E800000, 257)  # up to 2^126
    check(0, 65536, 1)
    check(0x7E800000 - 65536, 0x7E800000, 1)
