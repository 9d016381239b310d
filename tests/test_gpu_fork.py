"""The nonlocal chain beside the plane stage, from 8e5 grid points times pairs
on with the digit GEMMs and 6e6 with the FP64 one, and the digit passes and the
kinetic sum beside the projections, from 1e6 values on.  While kernels are timed
one by one, and once the stream was given a priority, they run in turn on one
stream: the same kernels on the same data, so every result is equal bit for bit,
also replayed from a graph.  Each test checks which of the two ran by the
context's count of work queued on its second stream."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ctx(pkg, s, prec, nmax):
    ctx = pkg.Context(*s["grid"], s["ka"], s["kb"], s["kc"], s["hmat"], precision=prec, max_states=nmax)
    ctx.set_vks(s["vks"])
    ctx.set_kb(s["kb_desc"])
    return ctx


def _timed(ctx, f):
    """f() with the kernels timed one by one, which keeps them on one stream."""
    n = ctx.side_runs
    ctx.set_timing(True)
    out = f()
    ctx.read_timing()
    ctx.set_timing(False)
    assert ctx.side_runs == n
    return out


# 48^3: 1.1e5 points a pair; contexts of 27 and more orbitals project with digit
# GEMMs, beside from 8 pairs on, the others and FP64 from 55 on
@pytest.mark.parametrize("prec,nmax,ns", [(0, 28, 28), (0, 108, 108), (0, 109, 109), (0, 130, 130), (1, 26, 26),
                                          (1, 28, 14), (1, 28, 15), (1, 28, 28), (1, 109, 109), (1, 130, 130),
                                          (2, 130, 130)])
def test_results_do_not_depend_on_the_streams(pkg, sys2, prec, nmax, ns):
    ctx = _ctx(pkg, sys2, prec, nmax)
    assert ctx.digit_gemms == (prec != 0 and nmax >= 27)
    beside = (ns + 1) // 2 * 48 ** 3 >= (8e5 if ctx.digit_gemms else 6e6)
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

    def equal(out):
        assert len(out) == len(ref)
        for a, b in zip(out, ref):
            assert np.array_equal(a, b)

    ref = _timed(ctx, results)
    for _ in range(3):
        n = ctx.side_runs
        equal(results())
        assert (ctx.side_runs > n) == beside
    n = ctx.side_runs
    b = pkg.Batch([ctx], [ns], [ec.size], [ec], [scale], [mean], [1.0])
    assert (ctx.side_runs > n) == beside
    for _ in range(2):
        b.launch()
        b.sync()
        assert np.array_equal(ctx.download_density(), ref[-1])
    b.close()
    n = ctx.side_runs
    for priority in (-2, 0):  # either marks the context as one of several at work
        ctx.sync()
        ctx.set_priority(priority)
        equal(results())
    assert ctx.side_runs == n
    ctx.close()


@pytest.mark.parametrize("prec,ns", [(0, 109), (1, 28)])
def test_a_graph_may_be_the_first_use_of_the_second_stream(pkg, sys2, prec, ns):
    """The second stream comes with the projectors, so that the capture of a
    one-context graph may be its first use; noise alone does not use it, nor does
    a context without projectors."""
    scale, mean, ec = 0.1, 2.0, 1.0 / np.arange(1.0, 10.0)
    ctx = _ctx(pkg, sys2, prec, ns)
    ctx.noise_dev(ns, seed=3.0)
    assert ctx.side_runs == 0
    b = pkg.Batch([ctx], [ns], [ec.size], [ec], [scale], [mean], [1.0])
    assert ctx.side_runs == ec.size - 1
    b.launch()
    b.sync()
    got = ctx.download_density()
    b.close()
    ctx.set_timing(True)  # in turn
    ctx.filter_cheby_dev(ns, ec, 1, scale, mean)
    assert np.array_equal(ctx.density_dev(ns), got)
    ctx.set_timing(False)
    n = ctx.side_runs
    ctx.set_kb(None)
    ctx.filter_cheby_dev(ns, ec, 1, scale, mean)
    assert ctx.side_runs == n
    ctx.set_kb(sys2["kb_desc"])
    ctx.filter_cheby_dev(ns, ec, 1, scale, mean)
    assert ctx.side_runs == n + ec.size - 1 and np.array_equal(ctx.density_dev(ns), got)
    ctx.close()


def test_lanczos_of_512_atoms_does_not_depend_on_the_streams(pkg, wl):
    """One orbital of 96^3, the smallest application that runs beside."""
    ctx = _ctx(pkg, wl.make_system(4, (96, 96, 96)), pkg.SDFT_PREC_MIXED, 1)
    ref = _timed(ctx, lambda: ctx.lanczos_bounds(12))
    for _ in range(2):
        n = ctx.side_runs
        out = ctx.lanczos_bounds(12)
        assert ctx.side_runs == n + 12
        assert out[:2] == ref[:2] and np.array_equal(out[2], ref[2]) and np.array_equal(out[3], ref[3])
    ctx.close()


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("ns", [60, 96, 330])  # 0.8e6 values of c in turn, 1.3e6 and 4.3e6 beside
def test_energies_and_forces_do_not_depend_on_the_streams(pkg, sys2, prec, ns):
    ctx = _ctx(pkg, sys2, prec, ns)
    ctx.noise_dev(ns, seed=5.0)
    ctx.filter_cheby_dev(ns, np.array([1.0, 0.5, 0.25]), 1, 0.1, 2.0)

    def results():
        f, e = ctx.nl_force_dev(ns)
        return [np.array(ctx.energy_chempot_dev(ns)), f, np.array(e)]

    ref = _timed(ctx, results)
    assert np.abs(ref[1]).max() > 0
    for _ in range(3):
        n = ctx.side_runs
        for a, b in zip(results(), ref):
            assert np.array_equal(a, b)
        # the kinetic sum, and with digit GEMMs three digit passes of the forces
        assert ctx.side_runs - n == (0 if ns == 60 else 4 if ctx.digit_gemms else 1)
    ctx.close()
