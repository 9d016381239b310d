"""Measured cases of the stochastic-DFT filter path.

Each case is one call (or one short sequence of calls) of this package's
public entry points on a seeded diamond-Si supercell: Gaussian local
potential, Gaussian s + p Kleinman-Bylander projectors, plane waves up to
10 Ha, ``nrep`` conventional 8-atom cells per axis.  What the kinds stand for
in real use:

  hpsi       one H psi on host buffers (calcCoefForceWrapSCF as PINY calls it)
  newton     a Newton filter on host buffers (filterNewtonPolyHerm)
  cheby      a Chebyshev filter; ``api`` "host": on host buffers, as
             filterChebyPolyHerm is called, with the moments it stores;
             "dev": resident orbitals, then the density of each chemical
             potential left on the device (the SCF step's form)
  moments    Chebyshev moments of resident orbitals (calcChebyMoments), once
             per SCF step before the chemical potential
  lanczos    the spectral range of H (20 Lanczos steps, one orbital)
  forces     energies and nonlocal atomic forces of filtered orbitals
  potential  V_KS from the density (cpGetVksStodft) on the density grid
  batch      several uneven systems, filters + densities as one graph

Grids: 24 points per cell and axis (the benchmark configurations), the grid
that holds the density sphere (32 per cell: PINY's own choice, and what a
filter that takes V_KS straight from ``potential`` runs on), or another
2^a 3^b edge of the same resolution.  Precision: 0 = FP64 (the default of
Context), 1 = mixed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__ as _entry

pkg = _entry.load_package()
wl = _entry.load_workload()

FP64, MIXED = 0, 1
EMIN, EMAX = -6.0, 11.5  # bounds of H for these cells: V in [-4.1, 0], 10 Ha cutoff, |E_KB| = 0.5
BETA = wl.BETA
OCC = wl.OCC


def _case(name, kind, rep, grid, nsto=0, order=0, prec=MIXED, nmu=1, api="dev", strain=(0.0, 0.0, 0.0), **more):
    c = {"kind": kind, "r1": rep[0], "r2": rep[1], "r3": rep[2], "n1": grid[0], "n2": grid[1], "n3": grid[2],
         "nsto": nsto, "order": order, "prec": prec, "nmu": nmu, "api": api,
         "e1": strain[0], "e2": strain[1], "e3": strain[2]}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one H psi of an orbital pair of 8 atoms
        _case("hpsi_8at_2orb", "hpsi", (1, 1, 1), (24, 24, 24), 2, 1, FP64, api="host"),
        # config 1: 8 atoms, 16 orbitals, Newton order 64, FP64, host buffers
        _case("newton_8at_16orb", "newton", (1, 1, 1), (24, 24, 24), 16, 64, FP64, api="host"),
        # config 2's system: 64 atoms, 48^3, 128 orbitals, resident, filter + density
        _case("cheby_64at_128orb", "cheby", (2, 2, 2), (48, 48, 48), 128, 64),
        # config 3's system: 512 atoms, 96^3, 512 orbitals, resident, filter + density
        _case("cheby_512at_512orb", "cheby", (4, 4, 4), (96, 96, 96), 512, 32),
        # 64 atoms on the density grid, two chemical potentials, an odd orbital count
        _case("cheby_64at_dgrid_97orb", "cheby", (2, 2, 2), (64, 64, 64), 97, 48, nmu=2),
        # an uneven strained cell on host buffers with moments (the drop-in call)
        _case("cheby_48at_uneven_host", "cheby", (3, 2, 1), (72, 48, 24), 131, 48, api="host",
              strain=(0.013, -0.017, 0.008)),
        # 216 atoms, 72^3 in FP64 (the default precision)
        _case("cheby_216at_fp64", "cheby", (3, 3, 3), (72, 72, 72), 64, 16, FP64),
        # moments for the chemical potential, 64 atoms on the density grid in FP64
        _case("moments_64at_dgrid_fp64", "moments", (2, 2, 2), (64, 64, 64), 48, 32, FP64),
        # spectral range of the 512-atom system
        _case("lanczos_512at", "lanczos", (4, 4, 4), (96, 96, 96), 1, 20),
        # energies and nonlocal forces of 512 atoms
        _case("forces_512at_256orb", "forces", (4, 4, 4), (96, 96, 96), 256, 2),
        # V_KS of 512 atoms on the density grid
        _case("potential_512at", "potential", (4, 4, 4), (128, 128, 128)),
        # six uneven systems (8 to 96 atoms) as one graph
        _case("batch_6_uneven", "batch", (2, 2, 3), (48, 48, 72), 96, 64, nsys=6, pick=4),
    ]


# ---------------------------------------------------------------------------
# drawn cases
# ---------------------------------------------------------------------------
def _edges(r, i, rng, how):
    """A grid edge for r cells: 24 per cell, the density grid's 32 per cell, or in between."""
    if how == "config":
        return 24 * r
    if how == "density":
        return 32 * r
    return {1: (24, 27, 32, 36), 2: (48, 54, 64), 3: (72, 81, 96), 4: (96, 108)}[r][rng.randrange(3 if r < 4 else 2)]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    top = work(listed()[3])["flops"]
    kinds = ("hpsi", "newton", "cheby", "cheby", "cheby", "moments", "lanczos", "forces", "potential", "batch")
    while True:
        kind = rng.choice(kinds)
        rep = tuple(rng.choice((1, 1, 2, 2, 3)) for _ in range(3)) if rng.random() < 0.85 else (4, 4, 4)
        if kind in ("batch", "newton", "hpsi") and rep == (4, 4, 4):
            rep = (2, 2, 2)
        how = rng.choice(("config", "config", "density", "other"))
        grid = tuple(_edges(r, i, rng, how) for i, r in enumerate(rep))
        strain = tuple(round(rng.uniform(-0.02, 0.02), 4) for _ in range(3))
        prec = rng.choice((FP64, MIXED, MIXED))
        c = _case(None, kind, rep, grid, _log(rng, 2, 512), _log(rng, 8, 128), prec, rng.choice((1, 1, 2)),
                  rng.choice(("dev", "host")), strain)
        if kind == "hpsi":
            c.update(nsto=_log(rng, 1, 64), order=1, nmu=1, api="host")
        elif kind == "newton":
            c.update(nsto=_log(rng, 2, 128), order=_log(rng, 8, 64), api="host")
        elif kind == "moments":
            c.update(order=2 * max(4, c["order"] // 2), nmu=1, api="dev")
        elif kind == "lanczos":
            c.update(nsto=1, order=20, nmu=1, api="dev")
        elif kind == "forces":
            c.update(order=2, nmu=1, api="dev")
        elif kind == "potential":
            g = wl.density_grid([wl.A0_SI * r * (1.0 + e) for r, e in zip(rep, strain)])
            c.update(n1=g[0], n2=g[1], n3=g[2], nsto=0, order=0, prec=FP64, nmu=1, api="dev")
            if max(g) > 128:
                continue
        elif kind == "batch":
            c.update(nsto=2 * max(8, c["nsto"] // 4), order=2 * max(8, c["order"] // 4), nmu=1, prec=MIXED, api="dev",
                     nsys=rng.randint(2, 8), pick=rng.randrange(1 << 16))
        if kind != "potential" and c["n1"] * c["n2"] > 96 * 128:
            continue  # planes past the library's shared-memory limit
        w = work(c)
        if w["flops"] > top * (0.1 if c["prec"] == FP64 else 1.0) or w["bytes"] > 4e9:
            continue
        return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _sphere(L, ecut):
    """Half sphere 0.5 |G|^2 <= ecut of an orthorhombic cell in PINY order, G = 0 last."""
    b = 2.0 * math.pi / np.asarray(L)
    m = [int(math.sqrt(2.0 * ecut) / x) + 1 for x in b]
    ka, kb, kc = np.meshgrid(np.arange(0, m[0] + 1), np.arange(-m[1], m[1] + 1), np.arange(-m[2], m[2] + 1),
                             indexing="ij")
    half = (ka > 0) | ((ka == 0) & ((kb > 0) | ((kb == 0) & (kc > 0))))
    keep = half & (0.5 * ((ka * b[0]) ** 2 + (kb * b[1]) ** 2 + (kc * b[2]) ** 2) <= ecut)
    return tuple(np.append(k[keep], 0).astype(np.int32) for k in (ka, kb, kc))


def _system(rep, grid, strain, seed, ecut=wl.ECUT_HA):
    sp = lambda hmat, e, kmax: _sphere(np.diag(hmat), e) + (None, None)  # noqa: E731
    return wl.make_system(rep, grid, strain=strain, disp_sigma=0.05, seed=seed, ecut=ecut, gvec=sp)


def _geometry(c):
    return (c["r1"], c["r2"], c["r3"]), (c["n1"], c["n2"], c["n3"]), (c["e1"], c["e2"], c["e3"])


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _maps(s, dev):
    n1, n2, n3 = s["grid"]
    ka, kb, kc = (torch.from_numpy(s[k].astype(np.int64)).to(dev) for k in ("ka", "kb", "kc"))
    at = lambda q: ((q * ka) % n1 * n2 + (q * kb) % n2) * n3 + (q * kc) % n3  # noqa: E731
    return at(1), at(-1)


def _noise(s, nsto, seed):
    """Noise orbitals: random +-1 on the grid, transformed to the sphere (complex [nsto, ncoef])."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    n1, n2, n3 = s["grid"]
    N = n1 * n2 * n3
    m, _ = _maps(s, dev)
    out = torch.empty(nsto, s["ncoef"], dtype=torch.complex128, device=dev)
    step = max(1, int(3e7) // N)
    for i in range(0, nsto, step):
        k = min(step, nsto - i)
        f = torch.randint(0, 2, (k, n1, n2, n3), generator=gen, device=dev, dtype=torch.int8).to(torch.float64) * 2 - 1
        out[i:i + k] = torch.fft.fftn(f, dim=(1, 2, 3)).reshape(k, N)[:, m] / math.sqrt(N)
    out[:, -1] = out[:, -1].real.to(torch.complex128)
    return out


def _host(z):
    z = z.reshape(-1)
    return z.real.contiguous().cpu().numpy(), z.imag.contiguous().cpu().numpy()


def _sqrt_fermi(e, mu):
    return np.sqrt(0.5 * (1.0 - np.tanh(np.clip(0.5 * BETA * (e - mu), -300, 300))))


def _cheby_coeffs(order, nmu):
    """a[k * nmu + imu]: Chebyshev coefficients of sqrt(Fermi) on [EMIN, EMAX]."""
    n = 32 * order
    th = math.pi * (np.arange(n) + 0.5) / n
    e = 0.5 * (EMIN + EMAX) + 0.5 * (EMAX - EMIN) * np.cos(th)
    cols = []
    for mu in (0.2, 0.35)[:nmu]:
        f = _sqrt_fermi(e, mu)
        a = np.array([2.0 / n * np.dot(f, np.cos(k * th)) for k in range(order)])
        a[0] *= 0.5
        cols.append(a)
    return np.stack(cols, axis=1).ravel()


def _newton(order, nmu):
    """Leja-ordered points on [-2, 2] and divided differences of sqrt(Fermi)."""
    scale = 4.0 / (EMAX - EMIN)
    cand = 2.0 * np.cos(math.pi * (np.arange(8 * order) + 0.5) / (8 * order))
    pts, d = [cand[0]], np.abs(cand - cand[0])
    logd = np.log(np.maximum(d, 1e-300))
    for _ in range(order - 1):
        i = int(np.argmax(logd))
        pts.append(cand[i])
        logd = logd + np.log(np.maximum(np.abs(cand - cand[i]), 1e-300))
    z = np.array(pts)
    cols = []
    for mu in (0.2, 0.35)[:nmu]:
        a = _sqrt_fermi(z / scale + 0.5 * (EMIN + EMAX), mu)
        for j in range(1, order):
            a[j:] = (a[j:] - a[j - 1:-1]) / (z[j:] - z[:-j])
        cols.append(a)
    return np.stack(cols, axis=1).ravel(), z, scale


def _batch_specs(c, seed):
    """(rep, grid, strain, system seed, nsto, order) of each system: shapes, orbital counts and orders from the case."""
    r = np.random.default_rng(c["pick"])
    out = []
    for i in range(c["nsys"]):
        while True:
            rep = tuple(int(x) for x in r.integers(1, 4, size=3))
            if rep[0] * rep[1] * rep[2] <= 12:
                break
        out.append((rep, tuple(24 * x for x in rep), tuple(float(x) for x in r.uniform(-0.02, 0.02, size=3)),
                    seed * 64 + i, 2 * int(r.integers(4, c["nsto"] // 2 + 1)), 2 * int(r.integers(4, c["order"] // 2 + 1))))
    return out


def _density_input(s, seed):
    """A positive density times the cell volume on the grid (package layout, a fastest)."""
    rng = np.random.default_rng(seed + 7)
    n1, n2, n3 = s["grid"]
    g = -s["vks"].reshape(n1, n2, n3)
    rho = g * (1.0 + 0.2 * rng.random((n1, n2, n3))) + 0.05
    vol = float(np.prod(s["L"]))
    rho *= s["num_elec"] / (rho.mean() * vol)
    return np.ascontiguousarray(rho.transpose(2, 1, 0).reshape(-1)) * vol


def _context(s, prec, nsto):
    ctx = pkg.Context(*s["grid"], s["ka"], s["kb"], s["kc"], s["hmat"], precision=prec, max_states=max(nsto, 1))
    ctx.set_vks(s["vks"])
    ctx.set_kb(s["kb_desc"])
    return ctx


def prepare(case, seed):
    c = case
    kind = c["kind"]
    rep, grid, strain = _geometry(c)
    st = {"c": c}
    if kind == "batch":
        ctxs, args = [], []
        for r, g, e, sd, nsto, order in _batch_specs(c, seed):
            s = _system(r, g, e, sd)
            ctx = _context(s, c["prec"], nsto)
            ctx.upload(*_host(_noise(s, nsto, sd)))
            ctxs.append(ctx)
            args.append((nsto, order, _cheby_coeffs(order, 1), OCC / nsto))
        n = len(ctxs)
        st["ctxs"] = ctxs
        st["batch"] = pkg.Batch(ctxs, [a[0] for a in args], [a[1] for a in args], [a[2] for a in args],
                                [2.0 / (EMAX - EMIN)] * n, [0.5 * (EMIN + EMAX)] * n, [a[3] for a in args])
        return st
    if kind == "potential":
        s = _system(rep, grid, strain, seed)
        dg = pkg.DensityGrid(*grid, s["hmat"], *_sphere(s["L"], 4.0 * wl.ECUT_HA))
        tab, gmin, d, g0 = wl.local_table()
        dg.set_local(s["pos"], tab, gmin, d, g0)
        st["grid"] = dg
        st["rho"] = torch.from_numpy(_density_input(s, seed)).to(_device())
        st["v"] = torch.empty(grid[0] * grid[1] * grid[2], dtype=torch.float64, device=_device())
        return st
    s = _system(rep, grid, strain, seed)
    ctx = st["ctx"] = _context(s, c["prec"], c["nsto"])
    if kind == "lanczos":
        rng = np.random.default_rng(seed)
        re, im = rng.standard_normal(s["ncoef"]), rng.standard_normal(s["ncoef"])
        im[-1] = 0.0
        st["v0"] = (re, im)
        return st
    re, im = _host(_noise(s, c["nsto"], seed))
    if kind in ("hpsi", "newton") or (kind == "cheby" and c["api"] == "host"):
        st["re"], st["im"] = re, im
    else:
        ctx.upload(re, im)
    if kind == "cheby":
        st["ec"] = _cheby_coeffs(c["order"], c["nmu"])
        if c["api"] == "dev":
            st["rho"] = torch.empty(c["nmu"], grid[0] * grid[1] * grid[2], dtype=torch.float64, device=_device())
    elif kind == "newton":
        st["ec"], st["samp"], st["scale"] = _newton(c["order"], c["nmu"])
    elif kind == "forces":  # orbitals as a short filter leaves them
        ctx.filter_cheby_dev(c["nsto"], _cheby_coeffs(c["order"], 1), 1, 2.0 / (EMAX - EMIN), 0.5 * (EMIN + EMAX))
        ctx.sync()
    return st


def run(state):
    c = state["c"]
    kind, ns = c["kind"], c["nsto"]
    scale, mean = 2.0 / (EMAX - EMIN), 0.5 * (EMIN + EMAX)
    if kind == "batch":
        state["batch"].launch()
        state["batch"].sync()
        return [ctx.download_density() for ctx in state["ctxs"]]
    if kind == "potential":
        _, gr, gi, e = state["grid"].vks_from_rho(state["rho"].data_ptr(), out_ptr=state["v"].data_ptr())
        return {"v": state["v"], "rho_g": (gr, gi), "energies": e}
    ctx = state["ctx"]
    if kind == "hpsi":
        fr, fi, e = ctx.calc_coef_force(state["re"], state["im"], want_enl=True)
        return {"force": (fr, fi), "enl": e}
    if kind == "newton":
        return ctx.filterNewtonPolyHerm(state["re"], state["im"], state["ec"], state["samp"], c["nmu"], state["scale"],
                                        mean)
    if kind == "cheby":
        if c["api"] == "host":
            return ctx.filterChebyPolyHerm(state["re"], state["im"], state["ec"], c["nmu"], scale, mean,
                                           store_moments=True)
        ctx.filter_cheby_dev(ns, state["ec"], c["nmu"], scale, mean)
        for k in range(c["nmu"]):
            ctx.density_dev(ns, imu=k, scale=OCC / ns, out_ptr=state["rho"][k].data_ptr())
        return state["rho"]
    if kind == "moments":
        return ctx.moments_dev(ns, c["order"], scale, mean)
    if kind == "lanczos":
        lo, hi, al, be = ctx.lanczos_bounds(nstep=c["order"], v0=state["v0"])
        return {"bounds": np.array([lo, hi]), "alpha": al, "beta": be}
    ek, ep = ctx.energy_chempot_dev(ns, occ=OCC)
    f, _ = ctx.nl_force_dev(ns, occ=OCC)
    return {"energies": np.array([ek, ep]), "force": f}


# ---------------------------------------------------------------------------
# work and tolerances
# ---------------------------------------------------------------------------
def _sizes(rep):
    """(half-sphere coefficients, KB projector rows) of a cell, to a few per cent."""
    atoms = 8 * rep[0] * rep[1] * rep[2]
    vol = atoms / 8.0 * wl.A0_SI ** 3
    ng = vol / (2.0 * math.pi) ** 3 * 4.0 / 3.0 * math.pi * (2.0 * wl.ECUT_HA) ** 1.5
    return 0.5 * ng, 4.0 * atoms


def _apply_flops(rep, grid):
    """Flops of one H psi of one orbital: KB projection and back projection, and two real transforms."""
    nc, p = _sizes(rep)
    N = grid[0] * grid[1] * grid[2]
    return 8.0 * p * nc + 5.0 * N * math.log2(N)


def work(case):
    c = case
    rep, grid, _ = _geometry(c)
    kind = c["kind"]
    nc, p = _sizes(rep)
    N = grid[0] * grid[1] * grid[2]
    vec = 16.0 * nc * c["nsto"]
    if kind == "batch":
        b = f = 0.0
        for r, g, _, _, nsto, order in _batch_specs(c, 0):
            n = g[0] * g[1] * g[2]
            b += 16.0 * _sizes(r)[0] * nsto + 16.0 * n
            f += nsto * ((order - 1) * _apply_flops(r, g) + 2.5 * n * math.log2(n))
        return {"bytes": b, "flops": f}
    if kind == "potential":
        return {"bytes": 16.0 * N + 8 * 24.0 * nc, "flops": 10.0 * N * math.log2(N)}
    one = c["nsto"] * _apply_flops(rep, grid)
    proj = 2 * 16.0 * p * nc
    if kind == "hpsi":
        return {"bytes": 2 * vec + 8.0 * N + proj, "flops": one}
    if kind in ("newton", "cheby"):
        rho = c["nmu"] if c["api"] == "dev" else 0
        out = rho * 8.0 * N if rho else c["nmu"] * vec
        return {"bytes": vec + out + 8.0 * N + proj,
                "flops": (c["order"] - 1) * one + rho * c["nsto"] * 2.5 * N * math.log2(N)}
    if kind == "moments":
        return {"bytes": vec + 8.0 * N + proj, "flops": (c["order"] // 2) * one}
    if kind == "lanczos":
        reads = c["order"] if proj > 1.2e8 else 1  # projectors larger than L2 are read by every step
        return {"bytes": reads * proj + 8.0 * N, "flops": c["order"] * one}
    return {"bytes": vec + 0.5 * proj, "flops": 16.0 * p * nc * c["nsto"]}


def tolerance(case):
    # about four times the largest difference from exact() over the listed
    # cases: 4.4e-7 in mixed precision (FP32 transforms, 28-bit projections),
    # 4.4e-12 in FP64 (the projectors' spline table against its formula)
    return {"rel": 2e-6} if case["prec"] == MIXED else {"rel": 2e-11}


# ---------------------------------------------------------------------------
# the same results in 64-bit torch
# ---------------------------------------------------------------------------
class _Ref:
    """H in complex128 on dense grids and dense projectors."""

    def __init__(self, s):
        self.s = s
        self.dev = _device()
        n1, n2, n3 = self.n = s["grid"]
        self.N = n1 * n2 * n3
        self.nc = s["ncoef"]
        self.map, self.mapc = _maps(s, self.dev)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(self.dev)  # noqa: E731
        self.v = t(s["vks"]).reshape(n1, n2, n3)
        b = 2.0 * math.pi / s["L"]
        self.g = torch.stack([t(s[k] * x) for k, x in zip(("ka", "kb", "kc"), b)], dim=1)
        self.g2 = (self.g ** 2).sum(1)
        self.vol = float(np.prod(s["L"]))
        self.step = max(1, int(4e7) // self.N)
        # projectors: row (atom, channel), complex, z = 2 Re sum_half conj(B) c for the l = 0
        # rows, and the same with B carrying the factor -i for l = 1
        rc, gg = wl.RC_KB, self.g2.sqrt()
        e = torch.exp(-0.5 * rc * rc * self.g2)
        n0 = math.sqrt(4.0 / (math.sqrt(math.pi) * rc ** 3))
        n_1 = math.sqrt(8.0 / (3.0 * math.sqrt(math.pi) * rc ** 5))
        f0 = 4.0 * math.pi * n0 * math.sqrt(math.pi / 2.0) * rc ** 3 * e * math.sqrt(1.0 / (4.0 * math.pi))
        f1 = 4.0 * math.pi * n_1 * math.sqrt(math.pi / 2.0) * rc ** 5 * gg * e * math.sqrt(3.0 / (4.0 * math.pi))
        y = self.g / torch.where(gg > 0, gg, torch.ones_like(gg))[:, None]
        ph = torch.exp(-1j * (t(s["pos"]) @ self.g.T))  # conj(e^{iGR})
        self.B = torch.cat([(ph * f0)[:, None]] + [(1j * ph * (f1 * y[:, d]))[:, None] for d in range(3)], dim=1)
        self.B = self.B.reshape(-1, self.nc)
        self.ekb = t(list(wl.EKB[:1]) + list(wl.EKB[1:]) * 3).repeat(len(s["pos"])) / self.vol

    def z(self, c):
        """KB projections [orbital, row] (real)."""
        w = c * 2.0
        w[:, -1] = c[:, -1]
        return w.real @ self.B.real.T + w.imag @ self.B.imag.T

    def real(self, c):
        """psi(r) [orbital, n1, n2, n3] of half-sphere coefficients."""
        k = c.shape[0]
        f = torch.zeros(k, self.N, dtype=torch.complex128, device=self.dev)
        f[:, self.mapc] = c.conj()
        f[:, self.map] = c
        return torch.fft.ifftn(f.reshape(k, *self.n), dim=(1, 2, 3), norm="forward").real

    def h(self, c, want_z=False):
        out = 0.5 * self.g2 * c
        z = self.z(c)
        w = z * self.ekb
        out += torch.complex(w @ self.B.real, w @ self.B.imag)
        for i in range(0, c.shape[0], self.step):
            f = torch.fft.fftn(self.real(c[i:i + self.step]) * self.v, dim=(1, 2, 3), norm="forward")
            out[i:i + self.step] += f.reshape(f.shape[0], self.N)[:, self.map]
        out[:, -1] = out[:, -1].real.to(torch.complex128)
        return (out, z) if want_z else out

    def density(self, c):
        rho = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        for i in range(0, c.shape[0], self.step):
            rho += (self.real(c[i:i + self.step]) ** 2).sum(0)
        return rho.permute(2, 1, 0).reshape(-1)

    @staticmethod
    def dot(a, b):
        """Per-orbital half-sphere inner products."""
        p = (a.conj() * b).real
        return 2.0 * p.sum(1) - p[:, -1]

    def cheby(self, chi, ec, order, nmu):
        """(filtered [nmu], sum over orbitals of <chi, T_k chi>)."""
        s, m = 2.0 / (EMAX - EMIN), 0.5 * (EMIN + EMAX)
        ec = ec.reshape(order, nmu)
        prev, cur = chi, s * (self.h(chi) - m * chi)
        acc = [ec[0, i] * chi + ec[1, i] * cur for i in range(nmu)]
        mom = [float(self.dot(chi, chi).sum()), float(self.dot(chi, cur).sum())]
        for k in range(2, order):
            prev, cur = cur, 2.0 * s * (self.h(cur) - m * cur) - prev
            for i in range(nmu):
                acc[i] += ec[k, i] * cur
            mom.append(float(self.dot(chi, cur).sum()))
        return acc, mom


def _xc(r):
    """Exchange potential, PZ81 correlation energy per particle and potential."""
    rs = (3.0 / (4.0 * math.pi * r)) ** (1.0 / 3.0)
    x = -(3.0 * r / math.pi) ** (1.0 / 3.0)
    q, ln = rs.sqrt(), rs.log()
    f1 = 1.0 + 1.0529 * q + 0.3334 * rs
    c_lo = -0.1423 / f1
    m_lo = c_lo * (1.0 + 7.0 / 6.0 * 1.0529 * q + 4.0 / 3.0 * 0.3334 * rs) / f1
    c_hi = 0.0311 * ln - 0.048 + 0.002 * rs * ln - 0.0116 * rs
    m_hi = 0.0311 * ln + (-0.048 - 0.0311 / 3.0) + 2.0 / 3.0 * 0.002 * rs * ln + (2.0 * -0.0116 - 0.002) / 3.0 * rs
    return x, torch.where(rs >= 1, c_lo, c_hi), torch.where(rs >= 1, m_lo, m_hi)


def _exact_potential(s, seed):
    dev = _device()
    n1, n2, n3 = s["grid"]
    N, vol = n1 * n2 * n3, float(np.prod(s["L"]))
    k = dict(zip(("ka", "kb", "kc"), _sphere(s["L"], 4.0 * wl.ECUT_HA)), grid=s["grid"])
    m, mc = _maps(k, dev)
    b = 2.0 * math.pi / s["L"]
    g = torch.stack([torch.from_numpy(k[q] * x) for q, x in zip(("ka", "kb", "kc"), b)], dim=1).to(dev)
    g2 = (g ** 2).sum(1)
    rho = torch.from_numpy(_density_input(s, seed)).to(dev).reshape(n3, n2, n1).permute(2, 1, 0)
    rg = torch.fft.fftn(rho, norm="forward").reshape(-1)[m]
    rg[-1] = rg[-1].real.to(torch.complex128)
    pos = torch.from_numpy(s["pos"]).to(dev)
    sf = torch.zeros_like(rg)
    for a in range(0, len(pos), 64):
        sf += torch.exp(-1j * (pos[a:a + 64] @ g.T)).sum(0)
    form = wl.V0_LOC * (2.0 * math.pi * wl.SIGMA_LOC ** 2) ** 1.5 * torch.exp(-0.5 * wl.SIGMA_LOC ** 2 * g2)
    vext = form * sf / vol
    gh = torch.where(g2 > 0, 4.0 * math.pi / (torch.where(g2 > 0, g2, torch.ones_like(g2)) * vol), torch.zeros_like(g2))
    eh = float((gh * (rg.abs() ** 2)).sum())
    ee = (vext.conj() * rg).real
    ee = float(2.0 * ee.sum() - ee[-1])
    vg = vext + gh * rg
    f = torch.zeros(N, dtype=torch.complex128, device=dev)
    f[mc] = vg.conj()
    f[m] = vg
    v = torch.fft.ifftn(f.reshape(n1, n2, n3), norm="forward").real
    r = rho / vol
    x, cc, mu = _xc(r)
    e = np.array([eh, ee, float((0.75 * x * r + cc * r).sum()) * vol / N, float(((x + mu) * r).sum()) * vol / N])
    return {"v": (v + x + mu).reshape(-1), "rho_g": _host(rg), "energies": e}


def exact(case, seed):
    c = case
    kind, ns = c["kind"], c["nsto"]
    rep, grid, strain = _geometry(c)
    if kind == "batch":
        out = []
        for r, g, e, sd, nsto, order in _batch_specs(c, seed):
            s = _system(r, g, e, sd)
            ref = _Ref(s)
            acc, _ = ref.cheby(_noise(s, nsto, sd), _cheby_coeffs(order, 1), order, 1)
            out.append((ref.density(acc[0]) * (OCC / nsto)).cpu().numpy())
        return out
    s = _system(rep, grid, strain, seed)
    if kind == "potential":
        return _exact_potential(s, seed)
    ref = _Ref(s)
    if kind == "lanczos":
        rng = np.random.default_rng(seed)
        v = torch.from_numpy(rng.standard_normal(s["ncoef"]) + 1j * rng.standard_normal(s["ncoef"])).to(ref.dev)[None]
        v[:, -1] = v[:, -1].real.to(torch.complex128)
        v = v / ref.dot(v, v).sqrt()
        p, b, al, be = torch.zeros_like(v), 0.0, [], []
        for _ in range(c["order"]):
            w = ref.h(v)
            a = float(ref.dot(v, w))
            w = w - a * v - b * p
            b = math.sqrt(max(float(ref.dot(w, w)), 0.0))
            al.append(a)
            be.append(b)
            p, v = v, w / b
        ev = np.linalg.eigvalsh(np.diag(al) + np.diag(be[:-1], 1) + np.diag(be[:-1], -1))
        return {"bounds": np.array([ev[0] - 0.1, ev[-1] + 0.1]), "alpha": np.array(al), "beta": np.array(be)}
    chi = _noise(s, ns, seed)
    if kind == "hpsi":
        h, z = ref.h(chi, want_z=True)
        f = -4.0 * h
        f[:, -1] *= 0.5
        return {"force": _host(f), "enl": float((ref.ekb * z * z).sum())}
    if kind == "newton":
        ec, samp, scale = _newton(c["order"], c["nmu"])
        ec = ec.reshape(c["order"], c["nmu"])
        cur, mean = chi, 0.5 * (EMIN + EMAX)
        acc = [ec[0, i] * chi for i in range(c["nmu"])]
        for k in range(1, c["order"]):
            cur = scale * ref.h(cur) - (scale * mean + samp[k - 1]) * cur
            for i in range(c["nmu"]):
                acc[i] += ec[k, i] * cur
        h = [_host(a) for a in acc]
        return [a for a, _ in h], [b for _, b in h]
    if kind == "cheby":
        acc, mom = ref.cheby(chi, _cheby_coeffs(c["order"], c["nmu"]), c["order"], c["nmu"])
        if c["api"] == "host":
            h = [_host(a) for a in acc]
            return [a for a, _ in h], [b for _, b in h], np.array(mom + [0.0])
        return torch.stack([ref.density(a) * (OCC / ns) for a in acc])
    if kind == "moments":  # <T_j, T_k> = (<T_{j+k}> + <T_{j-k}>) / 2 holds exactly in 64 bits too
        _, mom = ref.cheby(chi, np.zeros(c["order"] + 1), c["order"] + 1, 1)
        return np.array(mom)
    (a,), _ = ref.cheby(chi, _cheby_coeffs(c["order"], 1), c["order"], 1)
    z = ref.z(a)
    w = OCC / ns
    e = [w * float(ref.dot(a, 0.5 * ref.g2 * a).sum()), w * float((ref.ekb * z * z).sum())]
    f = torch.zeros(len(s["pos"]), 3, dtype=torch.float64, device=ref.dev)
    for d in range(3):
        dz = ref.z(1j * ref.g[:, d] * a)
        f[:, d] = -2.0 * w * (ref.ekb * z * dz).sum(0).reshape(-1, 4).sum(1)
    return {"energies": np.array(e), "force": f.cpu().numpy()}
