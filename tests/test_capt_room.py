"""The room that a tree built on the GPU takes for its lists: a build succeeds wherever the memory holds
twice what its largest level needs, the first guess too large for it or not."""
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
    text = "\n".join(f"{n} {limit} {len(needs)} " + " ".join(map(str, needs)) for n, limit, needs in cases)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout
    return [tuple(map(int, line.split())) for line in out.splitlines()]


def test_builds_that_fit_the_memory_succeed(tmp_path):
    rng = random.Random(5)
    cases = []
    for log in range(1, 31):
        leaves = 1 << log
        for _ in range(200):
            needs = [leaves]  # a level has at most twice the entries of the one before and one more a leaf
            while len(needs) < log:
                needs.append(int(needs[-1] * rng.uniform(0.9, 2.0)) + rng.randrange(leaves))
            # two levels' lists at a time, or two entries a leaf: four times the largest level does
            limit = int(4 * max(max(needs), leaves) * 2 ** rng.uniform(-3, 6))
            cases.append((leaves, limit, needs))
    for (leaves, limit, needs), (built, tried, guess) in zip(cases, _run(tmp_path, cases)):
        largest = max(max(needs), leaves)
        if limit >= 4 * largest:
            assert built == 1
        if limit < max(needs):
            assert built == 0
        # at most 8 smaller guesses, and one allocation a level
        assert tried <= 9 + len(needs)


def test_the_first_guess(tmp_path):
    # 160 entries a leaf, no less than 2^18, no more than 2^28 or two a leaf
    leaves = [2, 1024, 1 << 16, 1 << 21, 1 << 30]
    rows = _run(tmp_path, [(n, 1 << 62, [1, 1]) for n in leaves])
    assert [r[2] for r in rows] == [1 << 18, 1 << 18, 160 << 16, 1 << 28, 1 << 31]
    assert all(r[:2] == (1, 1) for r in rows)
