"""The room that a tree built on the GPU guesses for its lists: a build succeeds wherever the memory holds
what its levels need, the first guess too large for it or not, in a few attempts."""
import random
import shutil
import subprocess

import pytest

from conftest import ROOT


def _run(tmp_path, cases):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    exe = tmp_path / "capt_room_check"
    subprocess.run([gxx, "-O1", "-std=c++17", "-o", str(exe), str(ROOT / "tests" / "capt_room_check.cc")], check=True)
    text = "\n".join(" ".join(map(str, c)) for c in cases)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout
    return [tuple(map(int, line.split())) for line in out.splitlines()]


def test_builds_that_fit_the_memory_succeed(tmp_path):
    rng = random.Random(5)
    cases = []
    for log in range(1, 31):
        leaves = 1 << log
        for _ in range(200):
            needs = [int(leaves * 2 ** rng.uniform(-3, 11)) for _ in range(3)]
            limit = int(2 * max(max(needs), 2 * leaves) * 2 ** rng.uniform(-0.5, 8))
            cases.append((leaves, limit, *needs))
    for (leaves, limit, *needs), (built, attempts, entries) in zip(cases, _run(tmp_path, cases)):
        assert attempts < 16
        least = 2 * max(*needs, 2 * leaves)
        if limit >= least:
            assert built == 1 and entries >= max(needs) and 2 * entries <= limit
        if limit < 2 * max(needs):
            assert built == 0


def test_the_first_guess(tmp_path):
    # plenty of memory, small lists: 160 entries a leaf, no less than 2^18, no more than 2^28 or two a leaf
    leaves = [2, 1024, 1 << 16, 1 << 21, 1 << 30]
    rows = _run(tmp_path, [(n, 1 << 62, 1, 1, 1) for n in leaves])
    assert [r[2] for r in rows] == [1 << 18, 1 << 18, 160 << 16, 1 << 28, 1 << 31]
    assert all(r[:2] == (1, 1) for r in rows)
