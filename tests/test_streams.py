"""Executions of plans on several streams, from one thread and from several, share the device's work buffers: each
gives what it gives alone, to the bit.  So do the calls of a multi-electron object on streams of their own."""
import random
import threading

import numpy as np
import pytest

from tests.helpers import C0, C0PP, C1, PP, beamline, gaussian, make_wfr

torch = pytest.importorskip('torch')


def plans():
    from srw_b200.plan import Plan
    out = []
    for nx, ny, el, pp, sc in ((1024, 1024, C0, C0PP, {}), (1080, 900, C0, C0PP, {}),
                               (500, 490, C1, [PP(), PP(0, 1.25, 1.5, 1., 2.), PP(4)], dict(Rx=20., Ry=20., dRx=0.2, dRy=0.2))):
        ex, _, mesh = gaussian(nx, E=2012., sig=0.35e-3, r=1.5e-3, R=20., ny=ny)
        p = Plan(make_wfr(ex, 0.5j * ex, mesh, **sc), beamline(el, pp))
        ins = [torch.from_numpy(np.ascontiguousarray(a, np.complex64)).cuda() for a in (ex, 0.5j * ex)]
        ox, oy = p.new_output()
        p.execute(*ins, ox, oy)
        out.append((p, ins, ox, oy))
    torch.cuda.synchronize()
    return out


def run(p, ins, stream):
    with torch.cuda.stream(stream):
        ox, oy = p.new_output()
        p.execute(*ins, ox, oy)
    return ox, oy


@pytest.mark.gpu
@pytest.mark.parametrize('threads', [0, 6])
def test_streams_give_the_same_fields(threads):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    ref = plans()
    bad = []

    def work(k, streams, n):
        rng = random.Random(k)
        got = []
        for i in range(n):
            p, ins, ox, oy = ref[rng.randrange(len(ref))]
            got.append((run(p, ins, streams[i % len(streams)]), ox, oy))
            if i % 10 == 9:
                for s in streams:
                    s.synchronize()
                bad.extend(1 for g, x, y in got if not (torch.equal(g[0], x) and torch.equal(g[1], y)))
                got = []

    if threads == 0:
        work(1, [torch.cuda.Stream() for _ in range(4)], 60)
    else:
        ts = [threading.Thread(target=work, args=(k, [torch.cuda.Stream()], 30)) for k in range(threads)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    torch.cuda.synchronize()
    assert not bad, len(bad)


@pytest.mark.gpu
@pytest.mark.parametrize('graph', [False, True])
@pytest.mark.parametrize('rows', [120, 1500])                     # sampled rows, and all of them
def test_multi_electron_calls_on_several_streams(graph, rows):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from srw_b200.multie import MultiE, sample_offsets
    from srw_b200.plan import Plan
    sc = dict(Rx=20., Ry=20., dRx=0.2, dRy=0.2)
    ex, _, mesh = gaussian(500, E=2012., sig=0.35e-3, r=1.5e-3, R=20.)
    w, chain = make_wfr(ex, 0.5j * ex, mesh, **sc), beamline(C1, [PP(), PP(0, 2., 2., 2., 2.), PP(4)])
    m = Plan(w, chain).output_mesh()
    acc = dict(nx=100, ny=rows, eStart=mesh['eStart'], **{k: m[k] for k in ('xStart', 'xFin', 'yStart', 'yFin')})
    offs = sample_offsets(32, 30e-6, 5e-6, 5e-6, 2e-6, seed=3, sig_e=1e-3)
    got = []
    for n in (1, 4):
        streams = [torch.cuda.Stream() for _ in range(n)]
        me = MultiE(w, chain, acc, max_batch=4, graph=graph)
        for k in range(8):
            me.add(offs[4 * k:4 * k + 4], streams[k % n].cuda_stream)
        got.append(me.mean())                                     # on a stream of its own
        torch.cuda.synchronize()
    assert got[0].max() > 0 and np.array_equal(got[0], got[1])
