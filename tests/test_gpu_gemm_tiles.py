"""FP64 projection GEMMs over the orbital counts and splits at which the tile
shape, its remainders or the split of K change, against the CPU oracle; and
mixed contexts on both sides of the digit GEMMs' size limit.

FP64: sums of at most 1664 products in another order than the oracle's, 1e-12
as for every FP64 H psi.  Mixed: FP32 transforms and, above the limit, 28-bit
projections, 2e-7 as for every mixed H psi."""
import gc

import numpy as np
import pytest

from conftest import rel_l2
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _orbitals(nc, ns):
    rng = np.random.default_rng(ns)
    cr, ci = rng.standard_normal((ns, nc)), rng.standard_normal((ns, nc))
    ci[:, -1] = 0.0
    return cr.ravel(), ci.ravel()


def _ctx(pkg, s, prec, nmax):
    c = pkg.Context(*s["grid"], s["ka"], s["kb"], s["kc"], s["hmat"], precision=prec, max_states=nmax)
    c.set_vks(s["vks"])
    c.set_kb(s["kb_desc"])
    return c


def test_fp64_tiles_and_splits(pkg, sys1):
    o = O.OracleSys(sys1)
    ctx = _ctx(pkg, sys1, pkg.SDFT_PREC_FP64, 130)
    cr, ci = _orbitals(sys1["ncoef"], 130)
    nc = sys1["ncoef"]
    ref = np.concatenate([x.reshape(130, nc) for x in o.hpsi(cr, ci)], axis=1)
    for ns in (1, 7, 8, 9, 16, 17, 31, 33, 64, 65, 130):
        for split in (0, 1, 3, 13, 64):
            ctx.set_gemm_split(split)
            got = np.concatenate([x.reshape(ns, nc) for x in ctx.calc_coef_force(cr[:ns * nc], ci[:ns * nc])], axis=1)
            assert rel_l2(got, ref[:ns]) < 1e-12, (ns, split)
    ctx.close()


def test_fp64_tiles_of_a_larger_cell(pkg, wl):
    s = wl.make_system((2, 2, 1), (48, 48, 24), disp_sigma=0.05, seed=2)
    o = O.OracleSys(s)
    nc = s["ncoef"]
    cr, ci = _orbitals(nc, 40)
    ref = np.concatenate([x.reshape(3, nc) for x in o.hpsi(cr[:3 * nc], ci[:3 * nc])], axis=1)
    ctx = _ctx(pkg, s, pkg.SDFT_PREC_FP64, 40)
    for ns in (3, 20, 40):
        got = np.concatenate([x.reshape(ns, nc) for x in ctx.calc_coef_force(cr[:ns * nc], ci[:ns * nc])], axis=1)
        assert rel_l2(got[:3], ref) < 1e-12, ns
    ctx.close()


def test_fp64_split_of_more_orbitals_than_a_grid_dimension(pkg, wl):
    """A split projection of 65544 orbitals: the reduction's grid holds 65535 of
    them.  Eight orbitals repeated: every copy's force is the first one's, bit for
    bit (the same sums at another place), and equal to a context for eight."""
    s = wl.make_system(1, (12, 12, 12), ecut=5.0)
    nc, rep = s["ncoef"], 8193
    cr, ci = _orbitals(nc, 8)
    small = _ctx(pkg, s, pkg.SDFT_PREC_FP64, 8)
    ref = small.calc_coef_force(cr, ci)
    small.close()
    ctx = _ctx(pkg, s, pkg.SDFT_PREC_FP64, 8 * rep)
    ctx.set_gemm_split(3)
    got = ctx.calc_coef_force(np.tile(cr, rep), np.tile(ci, rep))
    ctx.close()
    for g, r in zip(got, ref):
        g = g.reshape(rep, 8 * nc)
        assert rel_l2(g[0], r) < 1e-12
        assert np.array_equal(g, np.broadcast_to(g[0], g.shape))


@pytest.mark.parametrize("nmax", [4, 1800])  # P K max_states = 2e5 and 9.6e7: DMMA and digit GEMMs
def test_mixed_on_both_sides_of_the_digit_limit(pkg, sys1, nmax):
    cr, ci = _orbitals(sys1["ncoef"], 4)
    ref = O.OracleSys(sys1).hpsi(cr, ci, want_enl=True)
    for prec, tol in ((pkg.SDFT_PREC_MIXED, 2e-7), (pkg.SDFT_PREC_MIXED_FAST, 6e-7)):
        ctx = _ctx(pkg, sys1, prec, nmax)
        fr, fi, e = ctx.calc_coef_force(cr, ci, want_enl=True)
        assert rel_l2(np.concatenate([fr, fi]), np.concatenate(ref[:2])) < tol
        assert abs(e - ref[2]) < 1e-6 * abs(ref[2])
        ctx.close()


@pytest.mark.parametrize("cells,grid,ns", [((2, 2, 2), (48, 48, 48), 2), ((3, 3, 3), (72, 72, 72), 2),
                                           ((3, 3, 3), (72, 72, 72), 4),  # FP64, FP64 and digit projectors
                                           ((2, 2, 2), (48, 48, 48), 256), ((3, 2, 1), (72, 48, 24), 96),
                                           ((4, 4, 4), (96, 96, 96), 512)])
def test_estimate_covers_either_form(pkg, wl, cells, grid, ns):
    """The admission estimate of a request covers all it allocates from the context
    to the density, set-up included, by no more than a tenth beside its fixed
    64 MB: under a limit of the estimate the calls succeed, under 0.9 of the rest
    one of them is refused its memory."""
    serve = __import__(pkg.__name__ + ".serve", fromlist=["estimate_bytes"])
    s = wl.make_system(cells, grid)
    est = serve.estimate_bytes(s, ns)

    gc.collect()  # contexts that earlier tests left would be released meanwhile

    def request(limit):
        pkg.set_device_memory_limit(0, pkg.device_memory_in_use(0) + int(limit))
        ctx = None
        try:
            ctx = _ctx(pkg, s, pkg.SDFT_PREC_MIXED, ns)
            ctx.lanczos_bounds(3)
            ctx.noise_dev(ns)
            ctx.moments_dev(ns, 4, 0.1, 2.0)
            ctx.filter_cheby_dev(ns, np.ones(3), 1, 0.1, 2.0)
            ctx.density_dev(ns, want=False)
            return ctx.device_bytes
        finally:
            pkg.set_device_memory_limit(0, 0)
            if ctx:
                ctx.close()

    assert request(est) <= est
    with pytest.raises(pkg.SdftError) as e:
        request(0.9 * (est - 64 * 2 ** 20))
    assert e.value.code == 3  # SDFT_ERR_NOMEM
