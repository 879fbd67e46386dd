"""The rule that takes a group's neighbour cells as one tile (vkfluidsim_gb300/csrc/vfs_tile_rule.h, the
functions that the kernels call), compiled for the host and compared with every cell's own key: a union
that is taken has distinct keys, and its runs are its cells' keys in visiting order; one that is refused
has two cells with one key, or lies at a wrap of the cells, of the hashes or (across a hash-block face)
of the table."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = tmp_path_factory.mktemp("tile_rule") / "check"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", f"-I{ROOT / 'vkfluidsim_gb300' / 'csrc'}",
                        str(ROOT / "tests" / "tile_rule" / "check.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(cases):
        text = "\n".join(" ".join(str(int(v)) for v in c) for c in cases)
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout
        got = np.array([ln.split() for ln in out.splitlines()], int).astype(bool)
        assert len(got) == len(cases)
        return got

    return run


SIZES = [1, 2, 9, 40, 700, 5110, 10_204, 10_205, 12_345, 65_536, 1_048_576, 4_613_734, 2**30]


@pytest.mark.parametrize("reach", [1, 2])
@pytest.mark.parametrize("where", ["inside", "faces", "wrap", "far", "small tables"])
def test_taken_unions_are_distinct_and_in_order(check, reach, where):
    rng = np.random.default_rng([reach, len(where)])
    cases = []
    for _ in range(4000):
        n = rng.choice(SIZES[:7] if where == "small tables" else SIZES)
        if where in ("inside", "small tables"):
            c = rng.integers(-15, 10, 3) + 50 * rng.integers(0, 40, 3)
        elif where == "faces":
            c = rng.integers(18, 27, 3) + 50 * rng.integers(-2, 4, 3)
        elif where == "wrap":  # cells whose cell + 25 wraps 2^32
            c = rng.integers(-36, -20, 3)
        else:
            c = rng.integers(-2**31, 2**31 - 16, 3)
        cases.append((reach, n, c[0] & 0xFFFFFFFF, (c[0] + rng.integers(0, 6)) & 0xFFFFFFFF, c[1] & 0xFFFFFFFF,
                      c[2] & 0xFFFFFFFF))
    taken, distinct, same = check(cases).T
    assert not np.any(taken & ~distinct) and not np.any(taken & ~same)
    assert taken.any() or where == "small tables"
    if where == "inside":  # one block and no wrap of the hashes: refused only for a shared key
        assert np.array_equal(taken, distinct)
    if where == "faces":  # (a table's end inside a row that crosses a face is refused too)
        assert np.mean(taken[distinct]) > 0.98


def test_runs_that_pass_the_end_of_the_table(check):
    """Rows whose keys reach n - 1 and continue at 0, at every place of the row."""
    cases = []
    for x in range(12):
        first = x + 50 * (7 + 50 * 9)  # the hash of cell (x - 25, 7 - 25, 9 - 25)
        for n in range(first - 2, first + 14):
            cases.append((2, n, (x + 2 - 25) & 0xFFFFFFFF, (x + 5 - 25) & 0xFFFFFFFF, 9 - 25 & 0xFFFFFFFF,
                          11 - 25 & 0xFFFFFFFF))
    taken, distinct, same = check(cases).T
    assert np.array_equal(taken, distinct) and np.array_equal(taken, same) and taken.any()
