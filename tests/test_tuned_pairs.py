"""The packaged launch shapes are ones the passes on pairs of lines launch: whole pairs, at most 512 threads of
their schedule's per CTA."""
import os
import re

from srw_b200 import tune

CSRC = os.path.join(os.path.dirname(tune.__file__), 'csrc')


def test_table_holds_whole_pairs():
    """(A shape of the earlier one-line passes, as columns of one pair at 2240 to 3840 points, made their column
    pass up to 1.7 times as long.)"""
    txt = open(os.path.join(CSRC, 'linep_lengths.h')).read()
    threads = {int(m[0]): int(m[1]) for m in re.findall(r'X\((\d+),[\d, ]*, (\d+)\)', txt)}
    rows = [l.split() for l in open(tune.TXT) if not l.startswith('#')]
    assert rows
    for axis, n, lines in ((f[0], int(f[1]), int(f[2])) for f in rows):
        assert lines % 2 == 0 and lines // 2 * threads[n] <= 512, (axis, n, lines)
        if axis == 'cols':
            assert lines >= 4 and lines & (lines - 1) == 0, (n, lines)      # 32-byte pieces of a row


def test_reported_lines_are_whole_pairs():
    """The lines per CTA that the library reports are those it launches: two per pair, also where an entry is odd."""
    import ctypes as C
    from srw_b200 import capi
    L = capi.lib()
    got = C.c_int()
    try:
        for axis, n, lines, want in ((0, 2240, 1, 2), (0, 2240, 2, 2), (0, 2240, 3, 2), (0, 512, 7, 6), (1, 512, 1, 2),
                                     (1, 512, 8, 8), (0, 2240, 0, 2), (1, 2240, 0, 4), (0, 4096, 0, 2), (1, 4096, 0, 4)):
            assert L.srwgTuneSetLines(axis, n, lines) == 0
            assert L.srwgTuneGetLines(axis, n, C.byref(got)) == 0
            assert got.value == want, (axis, n, lines)
    finally:
        L.srwgTuneLoad(tune.TXT.encode(), None)
