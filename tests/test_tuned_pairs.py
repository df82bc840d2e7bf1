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
