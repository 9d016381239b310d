"""Chebyshev moments on both sides of the number of partial sums up to which one
CTA adds them all: the moments of all orbitals against the sum over two subsets
whose partials it always adds.

Each moment is a combination of <chi|T_k chi>, <T_k chi|T_j chi> with factors of
at most 2, of magnitude at most |chi|^2 per orbital.  Two groupings differ by the
order of the sums (under 30 roundings, log2 of the terms) and, since the split
of the projections' sums follows the orbital count, in T_k itself: 11 roundings
a step (log2 of 1664 products), grown at most k^2 = 9 fold by the recurrence up
to T_3.  Under 2 (30 + 2 * 9 * 11) = 456 roundings of |chi|^2; 1000 are allowed,
where a lost partial sum would be 1 / 4098 of the whole."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [2, 3, 2730, 2731, 2742])  # 3 partials a pair at 24^3: 4095 and 4098 around the limit
def test_moments_add_up(pkg, sys1, ns):
    ctx = pkg.Context(*sys1["grid"], sys1["ka"], sys1["kb"], sys1["kc"], sys1["hmat"],
                      precision=pkg.SDFT_PREC_FP64, max_states=ns)
    ctx.set_vks(sys1["vks"])
    ctx.set_kb(sys1["kb_desc"])
    nc = sys1["ncoef"]
    rng = np.random.default_rng(ns)
    cr, ci = rng.standard_normal((ns, nc)), rng.standard_normal((ns, nc))
    ci[:, -1] = 0.0
    lo, hi = ctx.lanczos_bounds(20)[:2]
    scale, mean = 2.0 / (hi - lo), 0.5 * (hi + lo)
    m = ns // 2
    got = ctx.calcChebyMoments(cr.ravel(), ci.ravel(), 6, scale, mean)
    parts = [ctx.calcChebyMoments(cr[s].ravel(), ci[s].ravel(), 6, scale, mean) for s in (slice(0, m), slice(m, ns))]
    bound = 1000 * np.finfo(np.float64).eps * 2.0 * (np.sum(cr * cr) + np.sum(ci * ci))
    assert np.all(np.isfinite(got))
    assert np.max(np.abs(got - parts[0] - parts[1])) < bound
    ctx.close()
