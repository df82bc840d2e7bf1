"""The allocation-free entry point takes the chains that fit 1 MiB of tables, counted as factors per point: the
longest accepted and the first refused number of drifts on long, middle and square grids.  The accepted one
against the plan API, to the bit."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import PP, beamline, gaussian, make_wfr

torch = pytest.importorskip('torch')
ERR_STATIC_LIMIT = 23904


@pytest.mark.gpu
@pytest.mark.parametrize('nx,ny,most', [(8192, 32, 3), (2048, 128, 12), (512, 512, 24)])
def test_number_of_drifts_that_fit(nx, ny, most):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from srw_b200 import capi
    from srw_b200.plan import Plan
    from srw_b200.srwlpy import make_c_optc, make_c_wfr
    ex, _, mesh = gaussian(nx, E=1000., sig=100e-6, r=1e-3, ny=ny)
    ey = (0.3 + 0.2j) * ex
    w = make_wfr(ex, ey, mesh)
    dx, dy = (torch.from_numpy(np.ascontiguousarray(a, np.complex64)).cuda() for a in (ex, ey))
    for k in (most, most + 1):
        el = [e for i in range(k) for e in (('drift', 1. + 0.1 * i, 0), ('lens', 100., 100., 0., 0.))]
        chain = beamline(el, [PP()] * len(el))
        ox, oy = torch.zeros_like(dx), torch.zeros_like(dy)
        keep = []
        cw, co = make_c_wfr(w, keep), make_c_optc(chain, keep)
        r = capi.lib().srwgPropagElecFieldStatic(C.byref(cw), C.byref(co), dx.data_ptr(), dy.data_ptr(), ox.data_ptr(),
                                                 oy.data_ptr(), ox.numel(), None, None)
        torch.cuda.synchronize()
        if k > most:
            assert r == ERR_STATIC_LIMIT
            continue
        assert r == 0, capi.err_text(r)
        plan = Plan(w, chain)
        px, py = plan.new_output()
        plan.execute(dx, dy, px, py)
        torch.cuda.synchronize()
        assert float(px.abs().max()) > 0 and torch.equal(ox, px) and torch.equal(oy, py)
