"""Which host arrays of a mesh upload the GPU reads in place: only those that lie wholly inside the one pinned
range that holds their first byte. The rule, without a GPU; the arrays' addresses are numbers here."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
BASE, SIZE = 1 << 40, 1 << 20  # a registration, at the same address on the device


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    exe = tmp_path_factory.mktemp("pinned") / "pinned_range"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", f"-I{ROOT / 'axiomr_gb300' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "pinned_range.cpp"), "-o", str(exe)], check=True)

    def ask(host, bytes_, device=None, start=BASE, size=SIZE):
        line = f"{host} {host if device is None else device} {start} {size} {bytes_}\n"
        return int(subprocess.run([str(exe)], input=line, capture_output=True, text=True, check=True).stdout)

    return ask


@pytest.mark.parametrize("at,bytes_", [(0, 1), (0, SIZE), (16, SIZE - 16), (SIZE - 16, 16), (4096, 0)])
def test_inside(rule, at, bytes_):
    assert rule(BASE + at, bytes_) == BASE + at


@pytest.mark.parametrize("at,bytes_", [
    (0, SIZE + 1),            # only the front is pinned: one byte past the registration
    (0, 2 * SIZE), (16, SIZE), (SIZE - 16, 17), (SIZE - 4096, 1 << 30),
    (0, (1 << 64) - 1), (4096, (1 << 64) - 4096),  # a sum that wraps around
    (SIZE, 1), (SIZE + 16, 1)])  # past the range
def test_not_wholly_inside(rule, at, bytes_):
    assert rule(BASE + at, bytes_) == 0


def test_before_the_range(rule):
    assert rule(BASE - 16, 16) == 0 and rule(BASE - 16, 64) == 0


@pytest.mark.parametrize("off", [1, 4, 8, 12])
def test_unaligned(rule, off):
    assert rule(BASE + off, 64) == 0
    assert rule(BASE, 64, device=BASE + off) == 0


def test_unknown(rule):
    assert rule(BASE, 64, device=0) == 0           # ordinary memory
    assert rule(BASE, 64, start=0, size=0) == 0    # pinned, its range not known


def test_other_device_address(rule):
    there = 1 << 44
    assert rule(BASE + 32, 64, device=there + 32, start=there) == there + 32
    assert rule(BASE + 32, SIZE, device=there + 32, start=there) == 0
