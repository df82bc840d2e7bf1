"""Branches of the line passes that no other test reaches: a quartic angular phase of some radians (its sine and
cosine instead of its series), and lines of 16384 points (one line per thread) along either axis, against the
FP64 oracle.  Bars: five FP32 transforms come to about 5e-7 (14 instead of 6 to 10 doublings at 16384: 7e-7);
the factor of a phase of 3.5 rad adds its FP32 rounding (2e-7) and the hardware sine's 4e-7; a factor of four
is left."""
import numpy as np
import pytest

from tests.helpers import C0, C0PP, PP, beamline, gaussian, make_wfr, oracle_run, rel_l2

torch = pytest.importorskip('torch')


def check(ex, mesh, el, pp, sc, bar):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from srw_b200.plan import Plan
    rng = np.random.default_rng(ex.shape[1])
    ex = (ex * (1. + 0.3 * (rng.standard_normal(ex.shape) + 1j * rng.standard_normal(ex.shape)))).astype(np.complex64)
    ey = ((0.3 + 0.2j) * ex).astype(np.complex64)
    o = oracle_run(ex, ey, mesh, el, pp, **sc)
    plan = Plan(make_wfr(ex, ey, mesh, **sc), beamline(el, pp))
    ox, oy = plan.new_output()
    plan.execute(torch.from_numpy(ex).cuda(), torch.from_numpy(ey).cuda(), ox, oy)
    assert rel_l2(ox.cpu().numpy(), o.ex) < bar
    assert rel_l2(oy.cpu().numpy(), o.ey) < bar


@pytest.mark.gpu
@pytest.mark.parametrize('nx,ny', [(64, 64), (72, 90), (256, 128)])
def test_large_quartic_phase(nx, ny):
    # 100 eV, points 0.1 um apart: pi lam L q2 up to 1900 rad, the quartic phase up to 3.5 rad
    r = 0.5e-7 * (nx - 1), 0.5e-7 * (ny - 1)
    ex, _, mesh = gaussian(nx, E=100., sig=0.3 * r[0], r=r[0], ny=ny, ry=r[1])
    check(ex, mesh, [('drift', 1e-3, 0)], [PP()], {}, 4e-6)


@pytest.mark.gpu
@pytest.mark.parametrize('nx,ny', [(16384, 36), (36, 16384)])
def test_lines_of_16384_points(nx, ny):
    ex, _, mesh = gaussian(nx, E=2012., sig=0.35e-3, r=1.5e-3, R=20., ny=ny)
    check(ex, mesh, C0, C0PP, dict(Rx=20., Ry=20., dRx=0.2, dRy=0.2), 3e-6)
