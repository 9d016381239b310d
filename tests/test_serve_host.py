"""Host-side logic of the serving loop and the batch workload (no GPU):
request priorities, the device-memory estimate used for admission, the
seeded request stream and the uneven-system specs."""
import importlib

import numpy as np
import pytest


@pytest.fixture(scope="module")
def serve(pkg):
    return importlib.import_module(pkg.__name__ + ".serve")


def test_request_priority_orders_by_work(serve):
    small = serve.request_priority((24, 24, 24), 16, 128)
    mid = serve.request_priority((48, 48, 48), 128, 256)
    big = serve.request_priority((96, 96, 96), 256, 512)
    assert small <= mid <= big <= 0
    assert small == -5 and big == 0  # cheapest gets the most urgent level, 512 atoms the default


def test_memory_estimate_grows_with_work(serve, wl):
    specs = wl.batch_specs(nsys=12, seed=4, big_fraction=0.25)
    est = [serve.estimate_spec_bytes(s, s["nsto"]) for s in specs]
    assert all(e > 64 * 2 ** 20 for e in est)
    # more orbitals of the same system never need less memory
    s = specs[0]
    assert serve.estimate_spec_bytes(s, 2 * s["nsto"]) > serve.estimate_spec_bytes(s, s["nsto"])


def test_spec_estimate_close_to_built_estimate(serve, wl):
    # the pre-build estimate (cell volume and cutoff) brackets the exact one
    specs = wl.batch_specs(nsys=4, seed=9, big_fraction=0.0)
    for sp in specs:
        s = wl.build_spec(sp)
        exact = serve.estimate_bytes(s, sp["nsto"])
        pre = serve.estimate_spec_bytes(sp, sp["nsto"])
        assert 0.9 * exact <= pre <= 1.5 * exact


def test_poisson_requests_are_seeded_and_ordered(serve, wl):
    a = serve.poisson_requests(wl, 20, 50.0, seed=5, big_fraction=0.1)
    b = serve.poisson_requests(wl, 20, 50.0, seed=5, big_fraction=0.1)
    t = np.array([r["arrival"] for r in a])
    assert np.all(np.diff(t) > 0) and [r["seed"] for r in a] == [r["seed"] for r in b]
    assert [r["nsto"] for r in a] == [r["nsto"] for r in b]
    assert all(r["nsto"] % 2 == 0 and r["L"] % 2 == 0 for r in a)


def test_admission_refuses_what_never_fits(serve):
    gb = 1e9
    assert serve.admission(151 * gb, 0.0, 150 * gb, busy=False) == "refuse"
    assert serve.admission(151 * gb, 10 * gb, 150 * gb, busy=True) == "refuse"
    assert serve.admission(100 * gb, 60 * gb, 150 * gb, busy=True) == "wait"
    assert serve.admission(100 * gb, 60 * gb, 150 * gb, busy=False) == "admit"  # idle: whatever fits alone
    assert serve.admission(10 * gb, 60 * gb, 150 * gb, busy=True) == "admit"


def test_summary_counts_refused_and_failed(serve):
    rec = [dict(status="done", arrival=0.0, done=2.0, latency=2.0, nsto=16, phases={"x": 1.0}),
           dict(status="done", arrival=1.0, done=3.0, latency=2.0, nsto=32, phases={"x": 3.0}),
           dict(status="refused", arrival=1.5, nsto=256, L=512, reason="too big"),
           dict(status="failed", arrival=1.7, nsto=64, L=128, error="nomem", code=3)]
    s = serve.summarize(rec)
    assert (s["requests"], s["completed"], s["refused"], s["failed"]) == (4, 2, 1, 1)
    assert s["orbitals"] == 48 and abs(s["orbitals_per_s"] - 16.0) < 1e-12
    assert s["p50_ms"] == 2000.0 and s["prep_mean_s"] == {"x": 2.0}
    assert serve.summarize([rec[2]])["completed"] == 0


@pytest.mark.parametrize("mod", ["serve", "tuner"])
def test_serving_and_tuning_need_no_torch(pkg, mod):
    """The serving loop and the autotuner time and order device work through
    the library's own event calls: neither imports torch."""
    import ast
    import os
    src = open(os.path.join(os.path.dirname(pkg.__file__), mod + ".py")).read()
    names = set()
    for node in ast.walk(ast.parse(src)):
        if isinstance(node, ast.Import):
            names.update(a.name.split(".")[0] for a in node.names)
        elif isinstance(node, ast.ImportFrom) and node.module:
            names.add(node.module.split(".")[0])
    assert "torch" not in names


class _Ctx:
    """What the autotuner's cache key reads of a context, and the calls it makes."""
    n, precision = (48, 48, 48), 1

    def __init__(self, ncoef, max_states, digits):
        self.ncoef, self.max_states, self.digit_gemms, self.calls = ncoef, max_states, digits, []

    def set_gemm_bn(self, bn):
        self.calls.append(("bn", bn))

    def set_gemm_split(self, split):
        self.calls.append(("split", split))

    def set_plane_threads(self, nt):
        self.calls.append(("plane", nt))


def _tuner(pkg, path=None):
    mod = importlib.import_module(pkg.__name__ + ".tuner")
    t = mod.Tuner(pkg, path)
    t._time = lambda ctx, nstate, split, scale, emean: 1.0 if split in (0, 8) else 2.0
    return t


def test_tuned_shapes_are_kept_per_projection_gemm(pkg, tmp_path):
    """A split tuned on the digit GEMMs is not set on a context of the same grid
    and orbital tiles that projects with the FP64 GEMM, or the other way round;
    a file written before the key told them apart has no entry that matches."""
    import json
    digits, fp64 = _Ctx(6500, 40, True), _Ctx(6500, 20, False)
    t = _tuner(pkg)
    assert t.key(digits, 20, 256) != t.key(fp64, 20, 256)
    assert t.key(fp64, 20, 256) != t.key(_Ctx(6500, 200, False), 20, 256)  # more room for splits
    assert t.key(fp64, 20, 256) != t.key(_Ctx(13000, 20, False), 20, 256)  # twice the cutoff's K
    assert t.key(digits, 20, 256) == t.key(_Ctx(6500, 400, True), 20, 256)
    path = tmp_path / "shapes.json"
    path.write_text(json.dumps({"48x48x48/P256/N1/prec1": {"split": 32, "gemm_bn": 64}}))
    assert _tuner(pkg, str(path)).tune(fp64, 20, 256) == 0


def test_tile_widths_are_timed_for_digit_gemms_only(pkg):
    for digits in (True, False):
        ctx = _Ctx(6500, 40, digits)
        t = _tuner(pkg)
        t.tune(ctx, 40, 256)
        assert any(c[0] == "bn" for c in ctx.calls) == digits
        assert ("gemm_bn" in t.cache[t.key(ctx, 40, 256)]) == digits


@pytest.mark.parametrize("priorities,want", [(True, -5), (False, 0)])
def test_served_contexts_are_marked_as_several_at_work(serve, monkeypatch, priorities, want):
    """A context without a priority counts as alone on the device and takes a
    second stream, which slows the others' preparation: a server without stream
    priorities gives every context the default one."""
    class Stop(Exception):
        pass

    class Pkg:
        @staticmethod
        def set_device(device):
            pass

    class Wl:
        @staticmethod
        def build_spec(spec):
            return spec

    seen = []

    def prepare(*a, priority=None, **k):
        seen.append(priority)
        raise Stop

    monkeypatch.setattr(serve, "prepare", prepare)
    srv = serve.Server(Pkg, Wl, 1, priorities=priorities)
    with pytest.raises(Stop):
        srv._start(0, dict(spec=dict(grid=(24, 24, 24)), nsto=16, L=128, seed=1.0), 0.0)
    assert seen == [want]


def test_candidates_are_timed_as_replayed_graphs(pkg):
    """Not call by call, where a small system's launches by the host hide the shape."""
    log = []

    class Event:
        def __init__(self, device):
            pass

        def record(self, stream):
            log.append(("record", stream))

        def elapsed_ms(self, other):
            return 1.5

        def close(self):
            pass

    class Batch:
        stream_ptr = 7

        def __init__(self, ctxs, nstate, L, coeffs, scale, emean, occ):
            log.append(("graph", nstate[0], L[0], len(coeffs[0])))

        def launch(self):
            log.append("launch")

        def sync(self):
            log.append("sync")

        def close(self):
            log.append("close")

    class Pkg:
        pass

    Pkg.Event, Pkg.Batch = Event, Batch
    ctx = _Ctx(6500, 40, True)
    ctx.device = 0
    t = importlib.import_module(pkg.__name__ + ".tuner").Tuner(Pkg, steps=6)
    assert t._time(ctx, 40, 4, 0.1, 0.0, reps=1) == 1.5
    assert ctx.calls == [("split", 4)]
    assert log == [("graph", 40, 7, 7), "launch", ("record", 7), "launch", ("record", 7), "sync", "close"]
