"""The compile-time-edge FFT stages against the run-time-size ones (the same
library with SDFT_GENERIC_FFT=1 at context creation), over grids, precisions,
orbital counts and G lists, including one whose columns have gaps.

Both paths transform with the same arithmetic precision; FP64 results agree to
a few hundred roundings (1e-12), FP32 transforms (2^-24 per operation, about
30 operations deep and a handful of applications) to 5e-6."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


ECUT = {(12, 12, 12): 5.0, (24, 24, 32): 18.0}  # others 10 Ha


def _system(wl, grid, reps, holes, ecut=10.0):
    s = wl.make_system(reps, grid, strain=(0.01, -0.015, 0.005), disp_sigma=0.05, seed=3, ecut=ecut)
    if holes:  # drop interior points of some columns (the list stays grouped by column)
        drop = np.flatnonzero((s["kc"][:-1] == 1) & (s["kb"][:-1] % 3 == 1))
        assert len(drop)
        for k in ("ka", "kb", "kc"):
            s[k] = np.delete(s[k], drop)
        s["ncoef"] = len(s["ka"])
    return s


def _results(pkg, s, prec, ns, nmax=None, pairs=8):
    """Results of ns orbitals in a context for nmax, whose column stages take `pairs` column pairs a CTA."""
    ctx = pkg.Context(*s["grid"], s["ka"], s["kb"], s["kc"], s["hmat"], precision=prec, max_states=nmax or ns)
    assert ctx.column_pairs == pairs
    ctx.set_vks(s["vks"])
    ctx.set_kb(s["kb_desc"])
    out = {}
    cr, ci = ctx.genNoiseOrbitalReal(ns, seed=5.0)
    out["noise"] = np.concatenate([cr, ci])
    out["hpsi"] = np.concatenate(ctx.calc_coef_force(cr, ci))
    ec = np.linspace(1.0, 0.2, 14)
    sre, sim, mom = ctx.filterChebyPolyHerm(cr, ci, ec, 2, 2.0 / 17.5, 2.75, store_moments=True)
    out["filter"] = np.concatenate(sre + sim)
    out["stored moments"] = mom[:7]
    out["one mu"] = np.concatenate(sum(ctx.filterChebyPolyHerm(cr, ci, ec[:6], 1, 2.0 / 17.5, 2.75), []))
    out["newton"] = np.concatenate(sum(ctx.filterNewtonPolyHerm(cr, ci, ec[:5], np.linspace(-2, 2, 5), 1, 4.0 / 17.5,
                                                                2.75), []))
    out["moments"] = ctx.calcChebyMoments(cr, ci, 8, 2.0 / 17.5, 2.75)
    out["density"] = ctx.rhoCalcRealStoHybrid(cr, ci)
    ctx.close()
    return out


# every edge with a compile-time plan on every axis, the plane pairs with stage-B
# instances of their own, and spheres narrower and wider than 3/8 of the planes;
# the few orbitals make every context take the column stages of 8 pairs a CTA
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("grid,reps,ns,holes", [
    ((12, 12, 12), 1, 3, False), ((24, 24, 32), 1, 3, False), ((32, 32, 24), 1, 5, True),
    ((64, 64, 24), (2, 2, 1), 3, False), ((96, 64, 32), (3, 2, 1), 2, False), ((32, 96, 24), (1, 3, 1), 3, False),
    ((64, 32, 48), (2, 1, 2), 3, True), ((72, 48, 24), (3, 2, 1), 3, False), ((64, 96, 24), (2, 3, 1), 2, False),
    ((96, 32, 24), (3, 1, 1), 3, False), ((24, 24, 24), 1, 1, False), ((24, 24, 24), 1, 5, True),
    ((48, 24, 72), (2, 1, 3), 4, False), ((72, 72, 24), (3, 3, 1), 2, False), ((24, 72, 48), (1, 3, 2), 3, True),
    ((96, 96, 96), 2, 2, False), ((16, 18, 27), 1, 3, False), ((27, 16, 18), 1, 4, True), ((18, 27, 16), 1, 2, False),
    ((32, 36, 54), (1, 1, 2), 3, False), ((54, 32, 36), (2, 1, 1), 3, True), ((36, 64, 32), (1, 2, 1), 1, False),
    ((64, 54, 81), (2, 2, 3), 2, False), ((81, 64, 108), (2, 2, 3), 3, False), ((108, 81, 64), (3, 2, 2), 2, False),
    ((64, 108, 128), (2, 3, 3), 2, False), ((128, 48, 96), (3, 2, 3), 3, False), ((96, 128, 64), (3, 3, 2), 2, True)])
def test_compile_time_edges_match_run_time_sizes(pkg, wl, monkeypatch, prec, grid, reps, ns, holes):
    s = _system(wl, grid, reps, holes, ECUT.get(grid, 10.0))
    fast = _results(pkg, s, prec, ns)
    monkeypatch.setenv("SDFT_GENERIC_FFT", "1")
    slow = _results(pkg, s, prec, ns)
    for k, v in slow.items():
        assert rel_l2(fast[k], v) < (1e-12 if prec == 0 or k in ("noise", "density") else 5e-6), k


# the column stages of contexts with many orbitals: 32 column pairs a CTA below
# edge 36, 16 below 72 (43 and 87 column pairs here: the last CTA is partly empty)
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("grid,reps,ns,holes", [
    ((12, 12, 12), 1, 3, False), ((24, 24, 16), 1, 2, False), ((24, 24, 18), 1, 3, True), ((24, 24, 24), 1, 4, False),
    ((24, 24, 27), 1, 3, False), ((24, 24, 32), 1, 5, True), ((24, 24, 36), 1, 3, False),
    ((24, 24, 48), (1, 1, 2), 2, False), ((24, 24, 54), (1, 1, 2), 3, True), ((24, 24, 64), (1, 1, 2), 3, False)])
def test_columns_of_contexts_with_many_orbitals(pkg, wl, monkeypatch, prec, grid, reps, ns, holes):
    s = _system(wl, grid, reps, holes, ECUT.get(grid, 10.0))
    fast = _results(pkg, s, prec, ns, 1024, 32 if grid[2] < 36 else 16)
    monkeypatch.setenv("SDFT_GENERIC_FFT", "1")
    slow = _results(pkg, s, prec, ns)
    for k, v in slow.items():
        assert rel_l2(fast[k], v) < (1e-12 if prec == 0 or k in ("noise", "density") else 5e-6), k


# planes with an instance of their own and without one, most with 128 threads as
# the default: either CTA size can be set, and set back
@pytest.mark.parametrize("grid,reps", [((64, 64, 24), (2, 2, 1)), ((54, 64, 24), (2, 2, 1)), ((32, 32, 32), 1),
                                       ((32, 96, 24), (1, 3, 1)), ((108, 81, 32), (3, 2, 1))])
def test_plane_cta_sizes_give_the_same_result(pkg, wl, grid, reps):
    s = _system(wl, grid, reps, False)
    ctx = pkg.Context(*s["grid"], s["ka"], s["kb"], s["kc"], s["hmat"], precision=pkg.SDFT_PREC_MIXED, max_states=3)
    ctx.set_vks(s["vks"])
    ctx.set_kb(s["kb_desc"])
    cr, ci = ctx.genNoiseOrbitalReal(3, seed=5.0)
    ref = ctx.calc_coef_force(cr, ci)
    for nt in (256, 128, 0):
        ctx.set_plane_threads(nt)
        assert all(np.array_equal(a, b) for a, b in zip(ctx.calc_coef_force(cr, ci), ref)), nt
    ctx.close()
