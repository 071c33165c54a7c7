"""Host-side rules that pick a kernel's form, asked on the CPU through tests/cpp/launch_rules.cc."""
import os
import subprocess

import pytest

import pyb2vx as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
INT_MAX = 2 ** 31 - 1


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("rules") / "launch_rules")
    csrc = os.path.dirname(B.PRODUCT_LIB)
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-I" + csrc, "-I/usr/local/cuda/include",
                           os.path.join(ROOT, "tests", "cpp", "launch_rules.cc"), B.PRODUCT_LIB, "-Wl,-rpath," + csrc, "-o", exe])

    def answers(questions):
        out = subprocess.run([exe] + [",".join(str(f) for f in q) for q in questions], capture_output=True, text=True, timeout=60)
        assert out.returncode == 0, out.stderr
        return [tuple(int(f) for f in line.split()) for line in out.stdout.splitlines()]
    return answers


def test_rows_past_the_last_tile_do_not_wrap(ask):
    """In tiles of several pieces a row index runs up to five pieces past M before it is compared with it."""
    rows = [INT_MAX - d for d in (0, 1, 127, 128, 511, 512, 639, 640, 641, 100000)]
    for m, (pieces,) in zip(rows, ask([("pieces", m, 64, 148) for m in rows])):
        last_tile = (m - 1) // (128 * pieces) * (128 * pieces)
        assert pieces == 1 or last_tile + 127 + 128 * pieces <= INT_MAX, m
    assert ask([("pieces", INT_MAX - 640, 64, 148)]) == [(4,)]


def test_pieces_by_rows(ask):
    """Two tiles or more for each of four teams of every SM, and K up to 256."""
    one, two, four = 8 * 128 * 148, 2 * 8 * 128 * 148, 4 * 8 * 128 * 148
    rows = {1: 1, one: 1, two - 1: 1, two: 2, four - 1: 3, four: 4, 2 * four: 4}
    assert ask([("pieces", m, 256, 148) for m in rows]) == [(p,) for p in rows.values()]
    assert ask([("pieces", four, 272, 148), ("pieces", four // 2, 16, 74)]) == [(1,), (4,)]
