"""Lanczos steps past an invariant subspace: the device loop runs on, the call
cuts its result off at the vanishing beta.  Without projectors and with a
constant potential every plane wave is an eigenvector, so one step ends it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
def test_lanczos_stops_at_an_eigenvector(pkg, sys1, prec):
    s = sys1
    ctx = pkg.Context(*s["grid"], s["ka"], s["kb"], s["kc"], s["hmat"], precision=prec, max_states=3)
    ctx.set_vks(np.zeros(int(np.prod(s["grid"]))))
    v = np.zeros(s["ncoef"])
    v[5] = 1.0
    lo, hi, al, be = ctx.lanczos_bounds(nstep=8, v0=(v, np.zeros_like(v)))
    g = 2 * np.pi * np.array([s["ka"][5], s["kb"][5], s["kc"][5]]) / np.diag(s["hmat"])
    assert len(al) == len(be) == 1 and be[0] < 1e-12
    assert abs(al[0] - 0.5 * g @ g) < 1e-12 * al[0]
    assert lo == pytest.approx(al[0] - 0.1) and hi == pytest.approx(al[0] + 0.1)
    # the context serves later calls
    cr, ci = ctx.genNoiseOrbitalReal(3, seed=2.0)
    assert np.isfinite(ctx.calc_coef_force(cr, ci)[0]).all()
    ctx.close()
