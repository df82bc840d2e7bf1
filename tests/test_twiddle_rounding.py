"""Propagations between drifts of powers of two in 64 bits: no further off than with one table entry or the
product of two per twiddle factor.  Bars: what the earlier one-line-per-thread passes (16 x 4, 16 x 8, 16 x 16,
16 x 16 x 2, 16 x 16 x 4) were off on these inputs, their larger component, rounded up."""
import numpy as np
import pytest

from tests.helpers import C0, C0PP, beamline, gaussian, make_wfr, oracle_run, rel_l2

torch = pytest.importorskip('torch')


@pytest.mark.gpu
@pytest.mark.parametrize('n,bar', [(64, 3.4e-7), (128, 2.4e-7), (256, 4.3e-7), (512, 3.4e-7), (1024, 4.3e-7)])
def test_error_in_64_bits(n, bar):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from srw_b200.plan import Plan
    ex, _, mesh = gaussian(n, E=1000., sig=80e-6, r=1e-3)
    ex = ex.astype(np.complex64)
    ey = ((0.3 + 0.2j) * ex).astype(np.complex64)
    o = oracle_run(ex, ey, mesh, C0, C0PP)
    plan = Plan(make_wfr(ex, ey, mesh), beamline(C0, C0PP))
    ox, oy = plan.new_output()
    plan.execute(torch.from_numpy(ex).cuda(), torch.from_numpy(ey).cuda(), ox, oy)
    assert rel_l2(ox.cpu().numpy(), o.ex) < bar
    assert rel_l2(oy.cpu().numpy(), o.ey) < bar
