"""Shared-memory banks of the split lines and of the whole-array tiles (csrc/sj_split.cuh): the layouts are read
from the header, and every access pattern is counted over 32 banks of 4 bytes.  A 64-bit access is served per
half-warp, a 128-bit one per quarter-warp."""
import re
from pathlib import Path

import pytest

HEADER = (Path(__file__).resolve().parents[1] / "bridct_b200" / "csrc" / "sj_split.cuh").read_text()
CODE = re.sub(r"//[^\n]*", "", HEADER)


def _py(expr):
    """A C integer expression as Python."""
    expr = " ".join(expr.split()).replace("&&", " and ").replace("||", " or ")
    depth, q = 0, -1
    for i, ch in enumerate(expr):
        depth += {"(": 1, ")": -1}.get(ch, 0)
        if ch == "?" and depth == 0:
            q = i
            break
    if q >= 0:
        nest, depth = 0, 0
        for j in range(q + 1, len(expr)):
            depth += {"(": 1, ")": -1}.get(expr[j], 0)
            if depth == 0 and expr[j] == "?":
                nest += 1
            elif depth == 0 and expr[j] == ":":
                if nest == 0:
                    return f"(({_py(expr[q + 1:j])}) if ({_py(expr[:q])}) else ({_py(expr[j + 1:])}))"
                nest -= 1
    return expr.replace("/", "//")


def _grab(pattern):
    m = re.search(pattern, CODE, re.S)
    assert m, pattern
    return _py(m.group(1))


SPLIT = {int(n): (int(a), int(b)) for n, a, b in
         re.findall(r"struct Split<(\d+)> \{ static constexpr int A = (\d+), B = (\d+)", CODE)}
COL_PAIRS = _grab(r"constexpr int col_pairs\(\) \{ return (.*?); \}")
STRIP_ROW = _grab(r"int strip_row\(int r\) \{\s*return (.*?);\s*\}")
ROW_PITCH = _grab(r"struct RowGeo \{\s*static constexpr int P = (.*?);")
SWAPS = _grab(r"A = Split<N>::A, B = Split<N>::B, S = (.*?);\s*auto at")
SOURCE = _grab(r"int split_src\(int a, int b\) \{.*?return (.*?);")
TILE_PITCH = _grab(r"struct PairTileGeo \{.*?static constexpr int P = (.*?);")
ARRAY_PITCH = _grab(r"static constexpr int AP = (.*?);")


def _degree(addresses, words):
    """Largest number of different words of one bank among the lanes' accesses of `words` words."""
    banks = {}
    for a in addresses:
        assert a % words == 0
        for w in range(a, a + words):
            banks.setdefault(w % 32, set()).add(w)
    return max(len(s) for s in banks.values())


def _lanes(lp, warp, half, tasks):
    """(pair, task) of the 16 lanes of a half-warp; threads hold pair t % lp and task t / lp."""
    return [((32 * warp + 16 * half + k) % lp, ((32 * warp + 16 * half + k) // lp) % tasks) for k in range(16)]


def test_the_exchange_slots_are_the_ones_modelled():
    assert CODE.count("(b ^ (c % S)) * ES + (c * 2 + part) * (B * ES)") == 2
    assert CODE.count("((q % S) ^ (c % S)) * ES + (q - q % S) * ES") == 3   # == (q ^ (c % S)) * ES for a power of two S
    assert "e = ex(g) + c * (2 * B * ES)" in CODE


@pytest.mark.parametrize("n", sorted(SPLIT))
@pytest.mark.parametrize("rows", [False, True])
def test_exchange_of_a_split_line_has_no_conflicts(n, rows):
    a, b = SPLIT[n]
    lp = 8 if rows else eval(COL_PAIRS, {"N": n})
    s = eval(SWAPS, {"LP": lp})
    es = 2 * lp
    slot = lambda c, part, q: (c * 2 + part) * b * es + (q ^ (c % s)) * es
    for warp in range(4):
        for half in range(2):
            for part in range(2):
                for c in range(a // 2):      # stage 1: one column, the lanes' residues
                    assert _degree([slot(c, part, q) + 2 * p for p, q in _lanes(lp, warp, half, b)], 2) == 1
                for q in range(b):           # stage 2: one residue, the lanes' columns
                    assert _degree([slot(c, part, q) + 2 * p for p, c in _lanes(lp, warp, half, a // 2)], 2) == 1


@pytest.mark.parametrize("n", sorted(SPLIT))
def test_column_strips_have_no_conflicts(n):
    a, b = SPLIT[n]
    lp = eval(COL_PAIRS, {"N": n})
    at = lambda r, p: eval(STRIP_ROW, {"TC": 2 * lp, "r": r}) + 2 * p
    for half in range(2):
        for e in range(a):
            lanes = _lanes(lp, 0, half, b)
            assert _degree([at(eval(SOURCE, {"A": a, "B": b, "N": n, "a": e, "b": q}), p) for p, q in lanes], 2) == 1
        for k in range(0, n - 2, a):
            lanes = _lanes(lp, 0, half, a // 2)
            assert _degree([at(k + c, p) for p, c in lanes], 2) == 1


@pytest.mark.parametrize("n", sorted(SPLIT))
@pytest.mark.parametrize("lp", [8, 4])
def test_row_walks(n, lp):
    """Coefficients lie one apart for adjacent tasks: no conflicts.  Samples lie two apart (Makhoul's order): the
    lanes hit every other bank, twice."""
    a, b = SPLIT[n]
    pitch = eval(ROW_PITCH, {"N": n, "LP": lp})
    lanes = [(t % lp, t // lp) for t in range(32)]
    for k in range(0, n - 32 // lp, a):
        assert _degree([p * pitch + k + c for p, c in lanes], 1) == 1
    for e in range(a):
        src = lambda q: eval(SOURCE, {"A": a, "B": b, "N": n, "a": e, "b": q})
        assert _degree([p * pitch + src(q) for p, q in lanes], 1) == 2


@pytest.mark.parametrize("h,w", [(h, w) for h in (8, 16, 32, 64) for w in (8, 16, 32, 64) if h * w > 64])
def test_short_axes_of_tiles_have_no_conflicts(h, w):
    env = {"W": w, "H": h, "kRowPairs": 8}
    env["P"] = p = eval(TILE_PITCH, env)
    ap = eval(ARRAY_PITCH, env)
    pair = lambda l: l // (w // 2) * ap + 2 * (l % (w // 2))
    single = lambda l: l // w * ap + l % w
    row = lambda r: r // h * ap + r % h * p
    for i in range(h):
        assert _degree([pair(l) + i * p for l in range(16)], 2) == 1
        assert _degree([single(l) + i * p for l in range(32)], 1) == 1
    for first in range(0, 16, 8):
        assert _degree([row(first + l) for l in range(8)], 4) == 1
