"""Lengths with a fixed schedule of small radices (72 to 504), and the same rule's run-time schedules on
both sides of its limits (400 and 1600 points), along both axes, forward and backward, against the FP64
oracle.  Five FP32 transforms' roundings add up to about 5e-7: 3e-6 relative L2 leaves a factor of six."""
import numpy as np
import pytest

from tests.helpers import C0, C0PP, beamline, gaussian, make_wfr, oracle_run, rel_l2

torch = pytest.importorskip('torch')


@pytest.mark.gpu
@pytest.mark.parametrize('nx,ny', [(72, 504), (80, 432), (96, 392), (112, 360), (120, 336), (128, 288), (144, 280),
                                   (160, 256), (168, 240), (192, 224), (200, 216), (216, 200), (256, 128), (504, 72),
                                   (90, 100), (396, 420), (1560, 1620)])
def test_schedules_vs_oracle(nx, ny):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from srw_b200.plan import Plan
    ex, _, mesh = gaussian(nx, E=2012., sig=0.35e-3, r=1.5e-3, R=20., ny=ny)
    rng = np.random.default_rng(nx * 10000 + ny)
    noise = rng.standard_normal(ex.shape) + 1j * rng.standard_normal(ex.shape)
    ex = (ex * (1. + 0.1 * noise)).astype(np.complex64)
    ey = ((0.3 + 0.2j) * ex).astype(np.complex64)
    sc = dict(Rx=20., Ry=20., dRx=0.2, dRy=0.2, xc=0., yc=0.)
    o = oracle_run(ex, ey, mesh, C0, C0PP, **sc)
    w = make_wfr(ex, ey, mesh, **sc)
    plan = Plan(w, beamline(C0, C0PP))
    ox, oy = plan.new_output()
    plan.execute(torch.from_numpy(ex).cuda(), torch.from_numpy(ey).cuda(), ox, oy)
    assert rel_l2(ox.cpu().numpy(), o.ex) < 3e-6
    assert rel_l2(oy.cpu().numpy(), o.ey) < 3e-6
