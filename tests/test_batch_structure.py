"""Multi-electron runs whose detector rows lie about twice as far apart as the output's rows: the rule of
the sampled last pass (two output rows or more per detector row) then depends on the photon energy of each
electron.  The mean against the FP64 oracle run electron by electron, with replayed graphs and without;
its bar as in test_sampled_rows.py (FP32 transforms accurate to about 5e-7: 1e-5 leaves a factor of
ten)."""
import numpy as np
import pytest

from srw_b200.multie import sample_offsets
from tests.helpers import C1, PP, O, beamline, gaussian, make_wfr, rel_l2
from tests.test_multie import SIG, oracle_sum

torch = pytest.importorskip('torch')
SC = dict(Rx=20., Ry=20., dRx=0.2, dRy=0.2, xc=0., yc=0.)


def half_rows_case(n=12):
    """128 x 512 to 320 x 1280, a detector of half the rows over the same range (2.0016 output rows apart),
    electrons two by two on either side of the rule."""
    ex, _, mesh = gaussian(128, E=2012., sig=0.35e-3, r=1.5e-3, R=20., ny=512)
    ey = (0.3 + 0.2j) * ex
    pp = [PP(), PP(0, 1.25, 2., 1.25, 2.), PP(4)]
    o = O.Wfr.from_srwl(ex, ey, mesh, 20., 20., 0.2, 0.2, 0., 0.)
    O.propagate(o, [tuple(e) for e in C1], pp)
    m = o.out_mesh()
    assert (m['nx'], m['ny']) == (320, 1280)
    acc = dict(nx=96, ny=640, eStart=mesh['eStart'], **{k: m[k] for k in ('xStart', 'xFin', 'yStart', 'yFin')})
    offs = sample_offsets(n, *SIG, seed=5, sig_e=1e-3)
    offs[:, 4] = np.where(np.arange(n) // 2 % 2 == 0, -1e-3, 1e-3)
    return ex, ey, mesh, pp, acc, offs


def need_gpu():
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')


@pytest.mark.gpu
def test_graphs_of_mixed_electrons_vs_oracle():
    need_gpu()
    from srw_b200.multie import MultiE
    ex, ey, mesh, pp, acc, offs = half_rows_case()
    want = oracle_sum(dict(ex=ex, ey=ey, mesh=mesh), SC, C1, pp, acc, offs) / len(offs)
    assert np.abs(want).max() > 0
    w = make_wfr(ex, ey, mesh, **SC)
    for graph, batch in ((False, 4), (True, 1), (True, 2), (True, 4)):
        me = MultiE(w, beamline(C1, pp), acc, max_batch=batch, graph=graph)
        me.add(offs)
        assert me.count() == len(offs)
        assert rel_l2(me.mean(), want) < 1e-5, (graph, batch)


@pytest.mark.gpu
def test_mixed_electrons_run_as_one_batch():
    """A timed add refuses electrons that do not run as one batch."""
    need_gpu()
    from srw_b200.multie import MultiE
    ex, ey, mesh, pp, acc, offs = half_rows_case()
    me = MultiE(make_wfr(ex, ey, mesh, **SC), beamline(C1, pp), acc, max_batch=len(offs), graph=False)
    me.add_timed(offs)
    assert me.count() == len(offs)


@pytest.mark.gpu
@pytest.mark.parametrize('E,r,L,sx', [(806.7, 8e-3, 10., 30e-6), (440.4, 5e-5, 1e-2, 1e-6)])
def test_quartic_phase_at_its_limits(E, r, L, sx):
    """Angular drifts whose largest quartic phase, pi lam L q2 (lam^2 q2 / 4), lies at 2^-27 rad (below: left
    out) or 0.03 rad (below: by its series) and moves across with each electron's photon energy: one
    batch, to the same mean.  (The factor's error on either side is below its FP32 rounding.)"""
    need_gpu()
    from srw_b200.multie import MultiE
    ex, _, mesh = gaussian(512, E=E, sig=0.1 * r, r=r)
    ey = (0.3 + 0.2j) * ex
    sc = dict(Rx=0., Ry=0., dRx=0., dRy=0., xc=0., yc=0.)
    el, pp = [('drift', L, 0), ('lens', 1e3, 1e3, 0., 0.), ('drift', L, 0)], [PP()] * 3
    acc = dict(nx=64, ny=48, eStart=E, xStart=-0.8 * r, xFin=0.8 * r, yStart=-0.8 * r, yFin=0.8 * r)
    offs = sample_offsets(6, sx, 1e-6, sx, 1e-6, seed=5, sig_e=1e-3)
    offs[:, 4] = np.where(np.arange(6) % 2 == 0, 1e-3, -1e-3)
    want = oracle_sum(dict(ex=ex, ey=ey, mesh=mesh), sc, el, pp, acc, offs) / len(offs)
    assert np.abs(want).max() > 0
    me = MultiE(make_wfr(ex, ey, mesh, **sc), beamline(el, pp), acc, max_batch=len(offs), graph=False)
    me.add_timed(offs)
    assert me.count() == len(offs)
    assert rel_l2(me.mean(), want) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize('rows,n,graph', [(200, 66, False), (200, 40, False), (200, 66, True), (1600, 40, False),
                                          (1600, 66, True)])
def test_batches_in_parts_equal_whole_batches(rows, n, graph):
    """A batch whose work buffers would pass 8 GiB runs in parts (up to 66 electrons at 2048^2: 33 and 33, 40 of
    them 33 and 7), with sampled rows and with all of them: the same electrons in batches of 8 give the
    same sums up to the order of their FP64 additions (66 terms: 66 x 1.1e-16, a factor of ten left)."""
    need_gpu()
    from srw_b200.multie import MultiE
    from srw_b200.plan import Plan
    ex, _, mesh = gaussian(512, E=2012., sig=0.35e-3, r=1.5e-3, R=20.)
    ey = (0.3 + 0.2j) * ex
    pp = [PP(), PP(0, 2., 2., 2., 2.), PP(4)]
    w = make_wfr(ex, ey, mesh, **SC)
    m = Plan(w, beamline(C1, pp)).output_mesh()
    assert (m['nx'], m['ny']) == (2048, 2048)
    acc = dict(nx=100, ny=rows, eStart=mesh['eStart'], **{k: m[k] for k in ('xStart', 'xFin', 'yStart', 'yFin')})
    offs = sample_offsets(n, *SIG, seed=8, sig_e=1e-3)
    whole = MultiE(w, beamline(C1, pp), acc, max_batch=8, graph=False)
    whole.add(offs)
    want = whole.mean()
    del whole
    assert want.max() > 0
    parts = MultiE(w, beamline(C1, pp), acc, max_batch=66, graph=graph)
    for rep in range(4 if graph else 1):                         # both slots' graphs are captured, then replayed
        parts.reset()
        parts.add(offs)
        assert parts.count() == n
        np.testing.assert_allclose(parts.mean(), want, rtol=1e-13, atol=1e-13 * want.max())
    if not graph:
        parts.reset()
        assert all(v > 0 for v in parts.add_timed(offs))
        np.testing.assert_allclose(parts.mean(), want, rtol=1e-13, atol=1e-13 * want.max())
