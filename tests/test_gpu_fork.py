"""The nonlocal chain beside the plane stage, from 8e5 grid points times pairs
on with the digit GEMMs and 6e6 with the FP64 one, and the digit passes and the
kinetic sum beside the projections, from 1e6 values on.  While kernels are timed one by one, and once the stream has a
priority, they run in turn on one stream: the same kernels on the same data, so
every result is equal bit for bit, also replayed from a graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("ns", [26, 28, 108, 109, 130])  # 48^3: beside from 28 (digit GEMMs), 109 (FP64 GEMM)
def test_results_do_not_depend_on_the_streams(pkg, sys2, prec, ns):
    ctx = pkg.Context(*sys2["grid"], sys2["ka"], sys2["kb"], sys2["kc"], sys2["hmat"], precision=prec, max_states=ns)
    ctx.set_vks(sys2["vks"])
    ctx.set_kb(sys2["kb_desc"])
    lo, hi = ctx.lanczos_bounds(20)[:2]
    scale, mean = 2.0 / (hi - lo), 0.5 * (hi + lo)
    ec = 1.0 / np.arange(1.0, 10.0)

    def results():
        cr, ci = ctx.genNoiseOrbitalReal(ns, seed=3.0)
        out = [*ctx.calc_coef_force(cr, ci, want_enl=True), ctx.calcChebyMoments(cr, ci, 8, scale, mean)]
        (fr,), (fi,), m = ctx.filterChebyPolyHerm(cr, ci, ec, 1, scale, mean, store_moments=True)
        out += [fr, fi, m]
        ctx.noise_dev(ns, seed=3.0)
        ctx.filter_cheby_dev(ns, ec, 1, scale, mean)
        return out + [ctx.density_dev(ns)]

    ctx.set_timing(True)
    ref = results()
    ctx.read_timing()
    ctx.set_timing(False)
    for priority in (0, 0, -2):
        ctx.sync()
        ctx.set_priority(priority)
        for a, b in zip(results(), ref):
            assert np.array_equal(a, b)
    ctx.noise_dev(ns, seed=3.0)
    b = pkg.Batch([ctx], [ns], [ec.size], [ec], [scale], [mean], [1.0])
    for _ in range(2):
        b.launch()
        b.sync()
        assert np.array_equal(ctx.download_density(), ref[-1])
    b.close()
    ctx.close()


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("ns", [60, 96, 330])  # 0.8e6 values of c in turn, 1.3e6 and 4.3e6 beside
def test_energies_and_forces_do_not_depend_on_the_streams(pkg, sys2, prec, ns):
    ctx = pkg.Context(*sys2["grid"], sys2["ka"], sys2["kb"], sys2["kc"], sys2["hmat"], precision=prec, max_states=ns)
    ctx.set_vks(sys2["vks"])
    ctx.set_kb(sys2["kb_desc"])
    ctx.noise_dev(ns, seed=5.0)
    ctx.filter_cheby_dev(ns, np.array([1.0, 0.5, 0.25]), 1, 0.1, 2.0)

    def results():
        f, e = ctx.nl_force_dev(ns)
        return [np.array(ctx.energy_chempot_dev(ns)), f, np.array(e)]

    ctx.set_timing(True)
    ref = results()
    ctx.read_timing()
    ctx.set_timing(False)
    assert np.abs(ref[1]).max() > 0
    for _ in range(3):
        for a, b in zip(results(), ref):
            assert np.array_equal(a, b)
    ctx.close()
