"""Autotuner of the FFT line passes' launch shapes (the reference has none: FFTW plans per call,
gmfft.cpp:295; its CUDA build caches cuFFT plans, gmfft.h:182-187).

For every tuned line length (powers of two and the general lengths of csrc/linen_lengths.h) it times the
passes of an N x N propagation to the waist (a row pass and a column pass, the headline beamline's FFT) and of
an N x N drift (a column pass with two transforms between two row passes) for every valid number of lines
per CTA of each axis -- pairs of lines, so even numbers; it is also the CTA size and, for the column pass, the
width of the column blocks the row pass writes -- with CUDA events on the launching stream and L2 flushed
between repetitions.  Where the fastest pair of shapes beats the library's own
(about 256 threads, columns at least two pairs) by GAIN it goes into

  models/line_tuning.txt    "rows|cols N L" lines, read by the library at its first plan

and every measurement (ms per pass) into the file named by --json.  (models/line_tuning.json, which the
learned-factor cost model reads, holds the times of the one-line passes that came before those on pairs: the
choice of factors stays what the network was evaluated with.)

    python -m srw_b200.tune [--lengths 1280,2240] [--reps 15]          # GPU

torch supplies device memory, streams and events only.
"""
import argparse
import ctypes as C
import json
import os
import re
import time

import numpy as np

from . import capi

HERE = os.path.dirname(os.path.abspath(__file__))
TXT = os.path.join(HERE, 'models', 'line_tuning.txt')
JSN = os.path.join(HERE, 'models', 'line_tuning.json')
LENGTHS_H = os.path.join(HERE, 'csrc', 'linen_lengths.h')
SMEM_MAX = 220 * 1024
GAIN, STEP_MS = 0.02, 0.002           # a shape is worth an entry from 2 % and one step of the events' clock up


def general_lengths():
    txt = open(LENGTHS_H).read()
    block = txt[txt.index('SRWG_LINEN_LENGTHS(X)'):txt.index('SRWG_LINEN_POW2(X)')]
    return [int(v) for v in re.findall(r'X\((\d+)\)', block)]


def all_lengths(lo=256, hi=8192):
    p2 = [1 << k for k in range(8, 14) if lo <= (1 << k) <= hi]
    return sorted(set(p2 + [n for n in general_lengths() if lo <= n <= hi]))


def is_pow2(n):
    return n & (n - 1) == 0


FAM_POW2, FAM_SPEC = 1, 3          # classes of tuned lengths: powers of two, general lengths


def line_pitch(n, lines=1, cols=False):
    """The library's shared-memory pitch of a line (kernels.h line_pitch)."""
    p = n + n // 16
    r = (1 if lines >= 16 else 16 // lines) if (cols and lines >= 2) else 4
    return p + (r + 16 - p % 16) % 16
POW2_SPEC = [256, 512, 1024, 2048, 4096, 8192]       # powers of two whose entries may be of either class


def families(n):
    if is_pow2(n):
        return [FAM_POW2] + ([FAM_SPEC] if n in POW2_SPEC else [])
    return [FAM_SPEC]


def launch_shape(axis, n):
    """(class name, lines per CTA) of the line passes of n points along axis 0 (rows) or 1 (columns): 'pow2' or
    'spec' (a tuned general length) and the whole pairs of lines a CTA of the library takes, the tuning table's
    or its own choice; (None, 0) for other lengths.  (A launch of few lines takes fewer.)"""
    L = capi.lib()
    fam, lines = C.c_int(), C.c_int()
    capi.check(L.srwgTuneGetFamily(int(axis), int(n), C.byref(fam)), 'tune family')
    capi.check(L.srwgTuneGetLines(int(axis), int(n), C.byref(lines)), 'tune lines')
    name = {FAM_POW2: 'pow2', FAM_SPEC: 'spec'}.get(fam.value)
    return name, (lines.value if name else 0)


def pass_shapes(passes):
    """Launch shapes of the line passes of a plan (Plan.kernels() / MultiE.info() tuples)."""
    out = []
    for k in passes:
        if k[0] in ('line_rows', 'line_cols'):
            axis = 0 if k[0] == 'line_rows' else 1
            fam, lines = launch_shape(axis, k[1] if axis == 0 else k[2])
            out.append({"pass": "%s %dx%d" % (k[0], k[1], k[2]), "family": fam, "lines_per_cta": lines})
    return out


def candidates(axis, n, fam=None):
    """(class, lines per CTA) pairs the library's fixed_lines_valid accepts: shared memory, threads per CTA,
    columns a power of two up to 32; `fam` restricts them to one class (then plain lines per CTA are returned)."""
    out = []
    for f in families(n) if fam is None else [fam]:
        t = n // 16 if f == FAM_POW2 else (n + 15) // 16
        tmax = 1024 if f == FAM_POW2 else 512
        for L in range(1, 33):
            if L * line_pitch(n, L, axis == 1) * 8 > SMEM_MAX or t * L > tmax:
                break
            if axis == 1 and (L & (L - 1)):
                continue
            if axis == 0 and L > 8:
                break
            out.append(L if fam is not None else (f, L))
    return out


def _plan(n, dev, mode=4):
    """N x N Gaussian (2 keV, curved) through a 10 m drift to the waist: one row and one column pass; mode 0: by
    its angular representation, a column pass with two transforms between two row passes."""
    from . import srwlib as S
    from .plan import Plan
    r = 1.5e-3
    w = S.SRWLWfr()
    w.allocate(1, n, n)
    g = np.exp(-np.linspace(-r, r, n) ** 2 / (4. * (0.4e-3) ** 2))
    ex = (1e6 * g[:, None] * g).astype(np.complex64)
    a = np.empty(2 * n * n, np.float32)
    a[0::2], a[1::2] = ex.real.ravel(), ex.imag.ravel()
    w.arEx, w.arEy = a, a.copy()
    w.mesh.xStart, w.mesh.xFin, w.mesh.yStart, w.mesh.yFin = -r, r, -r, r
    w.mesh.eStart = w.mesh.eFin = 2012.
    w.Rx = w.Ry = 20.
    w.dRx = w.dRy = 0.2
    opt = S.SRWLOptC([S.SRWLOptD(10.)], [[0, 0, 1., mode, 0, 1., 1., 1., 1., 0, 0, 0]])
    return Plan(w, opt, device=dev.index), ex


def time_passes(n, rows, cols, dev, reps=15, flush=None):
    """CUDA-event time [ms] of the row and of the column passes of both chains with `rows` and `cols` lines per
    CTA (0: the library's own): the mean of the faster half of the repetitions (an event's time comes in steps
    of 2 us)."""
    import torch
    L = capi.lib()
    capi.check(L.srwgTuneSetLines(0, n, rows), 'tune rows')
    capi.check(L.srwgTuneSetLines(1, n, cols), 'tune cols')
    st = torch.cuda.current_stream(dev)
    t = {'line_rows': 0., 'line_cols': 0.}
    for mode, want in ((4, ['line_rows', 'line_cols']), (0, ['line_rows', 'line_cols', 'line_rows'])):
        p, ex = _plan(n, dev, mode)
        kinds = [k[0] for k in p.kernels()]
        if kinds != want:
            raise RuntimeError('unexpected passes %s' % kinds)
        a = torch.from_numpy(ex).to(dev)
        b = a.clone()
        ox, oy = p.new_output()
        for _ in range(2):
            p.execute(a, b, ox, oy)
        ms = []
        for _ in range(reps):
            if flush is not None:
                flush.fill_(1)
            ms.append(p.execute_timed(a, b, ox, oy, st))
        torch.cuda.synchronize(dev)
        m = np.sort(np.array(ms), 0)[:(reps + 1) // 2].mean(0)
        for k, v in zip(kinds, m):
            t[k] += float(v)
    return t['line_rows'], t['line_cols']


def tune(lengths, dev, reps=15, log=print, on_length=None):
    import torch
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)      # > L2 (126 MB)
    res = {}
    for n in lengths:
        t0 = time.time()
        even = [[L for L in candidates(axis, n, families(n)[0]) if L % 2 == 0] for axis in (0, 1)]
        dflt = time_passes(n, 0, 0, dev, reps, flush)
        meas = [(cr, cc) + time_passes(n, cr, cc, dev, reps, flush) for cc in even[1] for cr in even[0]]
        # of the shapes within 1 % of the fastest the one of fewest lines (a batch fills the chip anyway)
        fast = min((m[2] + m[3] for m in meas), default=0.)
        best = min((m for m in meas if m[2] + m[3] <= 1.01 * fast), key=lambda m: (m[0] + m[1], m[2] + m[3]), default=None)
        dflt = min(dflt, time_passes(n, 0, 0, dev, reps, flush), key=sum)
        if best is not None:                                           # again, beside the default
            again = time_passes(n, best[0], best[1], dev, reps, flush)
            need = max(GAIN * sum(dflt), STEP_MS)
            if sum(dflt) - (best[2] + best[3]) < need or sum(dflt) - sum(again) < need / 2:
                best = None
        res[n] = dict(rows=best[0] if best else 0, cols=best[1] if best else 0, rows_ms=best[2] if best else dflt[0],
                      cols_ms=best[3] if best else dflt[1], default_ms=list(dflt), measured=[list(m) for m in meas])
        log('N %5d  rows %2d %.4f ms  cols %2d %.4f ms  (default %.4f + %.4f ms)  %.1f s' % (
            n, res[n]['rows'], res[n]['rows_ms'], res[n]['cols'], res[n]['cols_ms'], dflt[0], dflt[1], time.time() - t0))
        for ax in (0, 1):
            capi.check(capi.lib().srwgTuneSetLines(ax, n, 0), 'tune')
        if on_length is not None:
            on_length(res)
    return res


def write(res, txt=TXT, jsn='', device_name=''):
    os.makedirs(os.path.dirname(txt) or '.', exist_ok=True)
    with open(txt, 'w') as f:
        f.write('# lines per CTA of the line passes on pairs where they beat the built-in choice by %g %% and 2 us or more, measured\n'
                '# by srw_b200.tune on %s (passes of an N x N propagation to the waist and of a drift, CUDA-event\n'
                '# time); lengths that are not listed run the built-in choice\n' % (100. * GAIN, device_name))
        for n in sorted(res):
            for ax in ('rows', 'cols'):
                if res[n][ax]:
                    f.write('%s %d %d\n' % (ax, n, res[n][ax]))
    if jsn:
        with open(jsn, 'w') as f:
            json.dump({'device': device_name, 'lengths': {str(n): res[n] for n in sorted(res)}}, f, indent=0)


def load_times(jsn=JSN):
    """{N: (rows ms, cols ms)} of the tuned launch shapes, or {} without a table."""
    if not os.path.exists(jsn):
        return {}
    d = json.load(open(jsn))
    return {int(n): (v['rows_ms'], v['cols_ms']) for n, v in d.get('lengths', {}).items()}


def main():
    import torch
    ap = argparse.ArgumentParser()
    ap.add_argument('--lengths', default='')
    ap.add_argument('--reps', type=int, default=15)
    ap.add_argument('--txt', default=TXT)
    ap.add_argument('--json', default='')
    args = ap.parse_args()
    dev = torch.device('cuda', 0)
    lengths = [int(v) for v in args.lengths.split(',') if v] or all_lengths()
    capi.lib().srwgTuneLoad(None, None)            # measure from the built-in defaults
    name = torch.cuda.get_device_name(dev)
    # the table is rewritten after every length, so that an interrupted run keeps what it measured
    res = tune(lengths, dev, args.reps, on_length=lambda r: write(r, args.txt, args.json, name))
    write(res, args.txt, args.json, name)
    print('wrote %s' % ', '.join(f for f in (args.txt, args.json) if f))


if __name__ == '__main__':
    main()
