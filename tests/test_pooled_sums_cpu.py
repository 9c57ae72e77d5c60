"""Where the prompt kernel of pooled attention reads and writes its sums: every group's walk stays in the unit's part of the workspace and
meets each of its places once (csrc/pooled_sums.h, built for the host)."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "amd-pace_b200", "csrc")
SOURCE = """#include "pooled_sums.h"
extern "C" int groups() { return pace::PooledSums::kGroups; }
extern "C" int size(int h, int p, int r) { return pace::PooledSums{h, p, r}.size(); }
extern "C" int first(int h, int p, int r, int g) { return pace::PooledSums{h, p, r}.first(g); }
extern "C" int next(int h, int p, int r, int g, int head, int piece, int round) { return pace::PooledSums{h, p, r}.next(g, head, piece, round); }
"""


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    d = tmp_path_factory.mktemp("sums")
    (d / "s.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "s.cpp"), "-o", str(d / "s.so")], check=True)
    return C.CDLL(str(d / "s.so"))


@pytest.mark.parametrize("heads", [1, 2, 3, 4])
@pytest.mark.parametrize("pieces", range(1, 9))
@pytest.mark.parametrize("rounds", [1, 2, 3])
def test_walks_stay_in_the_unit(sums, heads, pieces, rounds):
    shape, size = (heads, pieces, rounds), sums.size(heads, pieces, rounds)
    block = 4 * 128
    assert size == heads * pieces * rounds * block
    seen = []
    for g in range(sums.groups()):
        at = sums.first(*shape, g)                  # asked for by every group, whether it has a piece or not
        assert at == -1 or 0 <= at <= size - block
        assert (at == -1) == (g >= pieces)
        for head in range(heads):
            for piece in range(g, pieces, sums.groups()):
                for r in range(rounds):
                    assert at == ((head * pieces + piece) * rounds + r) * block     # what is worked on now was asked for
                    seen.append(at)
                    at = sums.next(*shape, g, head, piece, r)
                    assert at == -1 or 0 <= at <= size - block
        assert at == -1
    assert sorted(seen) == list(range(0, size, block))


def test_workspace_holds_every_unit():
    from pace_b200 import _C
    # (heads, KV heads, value elements): one unit of one tile; two KV heads of 16 elements have fewer pieces than there are groups
    for H, G, vdim, tile in ((2, 2, 16, 128), (3, 3, 16, 128), (4, 2, 16, 64), (8, 2, 48, 32), (10, 5, 120, 64)):
        n = _C.lib.pace_attn_pooled_prompt_workspace_bytes(1, tile, H, G, vdim, 1)
        parts = (32 // (H // G)) * ((H // G + 3) // 4) * 4
        assert n >= G * ((vdim + 15) // 16) * ((parts + 31) // 32) * 4 * 128 * 16
