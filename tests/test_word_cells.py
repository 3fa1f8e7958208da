"""The bound that sizes the sweep loop's candidate lists: the most cells of one
colour, (i + j + k) mod 3, in a word of 32 consecutive cells, with every cell of
the mesh fluid (a caller's flags are not checked for a frame).
"""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _word_cells():
    src = open(os.path.join(ROOT, "pdac_b200", "csrc", "inner.cuh")).read()
    return int(re.search(r"constexpr int WORD_CELLS = (\d+);", src).group(1))


def test_bound_for_any_mesh():
    """Rows of nx >= 5 cells whose residues are unrelated (a row's first cell
    may have any colour): w consecutive cells of a row hold at most
    ceil(w / 3) of one."""
    most = 0
    for nx in range(5, 130):
        for first in range(nx):  # the word starts in column `first` of a row
            total, left, lo = 0, 32, first
            while left:
                w = min(nx - lo, left)
                total += -(-w // 3)
                left -= w
                lo = 0
            most = max(most, total)
    assert most == _word_cells()


def test_words_of_small_meshes():
    worst = 0
    for nx in range(5, 14):
        for ny in (1, 5, 6, 7):
            for nz in (5, 6, 9, 20):
                n = nx * ny * nz
                colour = [(c % nx + c // nx % ny + c // (nx * ny)) % 3 for c in range(n)]
                for t in range(0, n, 32):
                    word = colour[t:t + 32]
                    worst = max(worst, *(word.count(q) for q in range(3)))
    assert 11 < worst <= _word_cells()
