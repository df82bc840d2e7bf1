"""Multi-electron batches whose last pass transforms only the rows the detector samples (a detector row
per two output rows or more), and the rule's other side, against the FP64 oracle run electron by electron:
detectors coarser and finer than the limit, beyond the electrons' meshes, of odd sizes and a few points;
lengths with and without a fixed schedule; batches in one and several parts.  The mean intensity is a
sum of squares of FP32 transforms accurate to about 5e-7: 1e-5 relative L2 leaves a factor of ten."""
import numpy as np
import pytest

from srw_b200.multie import sample_offsets
from tests.helpers import C1, PP, O, beamline, gaussian, make_wfr, rel_l2
from tests.test_multie import SIG, oracle_sum

torch = pytest.importorskip('torch')


@pytest.mark.gpu
@pytest.mark.parametrize('n,ny,fac,acc_n,span,batch', [
    (128, 128, (1.25, 2., 1.25, 2.), (96, 80), 0.9, 4),      # 320 x 320, about four output rows apart: sampled
    (128, 120, (1., 1.5, 1., 1.25), (41, 150), 1.3, 3),      # about the mesh's own rows: every row transformed
    (121, 97, (1.25, 1.5, 0.75, 2.), (33, 29), 1.2, 7),      # odd meshes, lengths without a fixed schedule
    (100, 90, (2., 2., 2., 2.), (2, 3), 0.5, 2),             # a detector of a few points
    (90, 100, (1.5, 1.75, 2., 1.), (700, 11), 2.5, 6),       # fine along x, coarse along y, mostly outside
])
def test_mean_intensity_vs_oracle(n, ny, fac, acc_n, span, batch):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from srw_b200.multie import MultiE
    ex, _, mesh = gaussian(n, E=2012., sig=0.35e-3, r=1.5e-3, R=20., ny=ny)
    ey = (0.3 + 0.2j) * ex
    sc = dict(Rx=20., Ry=20., dRx=0.2, dRy=0.2, xc=0., yc=0.)
    pp = [PP(), PP(0, *fac), PP(4)]
    o = O.Wfr.from_srwl(ex, ey, mesh, 20., 20., 0.2, 0.2, 0., 0.)
    O.propagate(o, [tuple(e) for e in C1], pp)
    m = o.out_mesh()
    acc = dict(nx=acc_n[0], ny=acc_n[1], eStart=mesh['eStart'], **{k: span * m[k] for k in ('xStart', 'xFin', 'yStart', 'yFin')})
    offs = sample_offsets(7, *SIG, seed=5, sig_e=1e-3)
    want = oracle_sum(dict(ex=ex, ey=ey, mesh=mesh), sc, C1, pp, acc, offs) / len(offs)
    assert np.abs(want).max() > 0
    w = make_wfr(ex, ey, mesh, **sc)
    for graph in (False, True):
        me = MultiE(w, beamline(C1, pp), acc, max_batch=batch, graph=graph)
        me.add(offs)
        assert me.count() == len(offs)
        assert rel_l2(me.mean(), want) < 1e-5
