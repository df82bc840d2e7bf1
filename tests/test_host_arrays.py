"""The entry point on host arrays against the same plan on device arrays, to the bit: fields below and
above the size that is copied by several threads, ragged last blocks, one component, arrays in pinned
memory."""
import numpy as np
import pytest

from tests.helpers import PP, beamline, gaussian, make_wfr

torch = pytest.importorskip('torch')
CHAIN = [('lens', 10., 10.), ('drift', 2., 0)]


@pytest.mark.gpu
@pytest.mark.parametrize('n,ny,fac,comps,pinned', [
    (64, 60, (1., 1., 1., 1.), 'xy', False),          # a few kB: one copy
    (512, 512, (1., 1., 1., 1.), 'xy', False),        # exactly the limit of 4 MiB, in and out
    (512, 504, (1., 1.5, 1., 1.), 'xy', False),       # in below it, out above
    (728, 702, (1., 1., 1., 1.), 'x', False),         # one component, a short last block
    (900, 1100, (1., 2., 1., 1.), 'xy', False),       # more blocks than the threads hold at once
    (900, 1100, (1., 1., 1., 1.), 'xy', True),        # pinned arrays: copied in place
])
def test_host_arrays_equal_device_arrays(n, ny, fac, comps, pinned):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from srw_b200 import srwlpy
    from srw_b200.plan import Plan
    ex, _, mesh = gaussian(n, E=2012., sig=0.35e-3, r=1.5e-3, R=20., ny=ny)
    rng = np.random.default_rng(n)
    ex = (ex * (1. + 0.1 * rng.standard_normal(ex.shape))).astype(np.complex64)
    ey = (0.3 + 0.2j) * ex if 'y' in comps else 0 * ex
    sc = dict(Rx=20., Ry=20., dRx=0.2, dRy=0.2, xc=0., yc=0.)
    chain = beamline(CHAIN, [PP(0, *fac), PP()])
    w = make_wfr(ex, ey, mesh, **sc)
    plan = Plan(w, chain)
    ox, oy = plan.new_output()
    dev = [torch.from_numpy(np.ascontiguousarray(a, np.complex64)).cuda() for a in (ex, ey)]
    plan.execute(dev[0], dev[1], ox, oy)
    want = [t.cpu().numpy() for t in (ox, oy)]
    for rep in range(2):                              # the second call meets the first one's blocks
        w = make_wfr(ex, ey, mesh, **sc)
        if 'y' not in comps:
            w.arEy = None
        hold = []
        if pinned:
            for c in ('arEx', 'arEy'):
                t = torch.from_numpy(getattr(w, c)).pin_memory()
                hold.append(t)
                setattr(w, c, t.numpy())
        srwlpy.PropagElecField(w, chain)
        assert np.array_equal(w.field('x').reshape(want[0].shape), want[0])
        if 'y' in comps:
            assert np.array_equal(w.field('y').reshape(want[1].shape), want[1])
