"""Host result arrays are not cleared before the call that fills them; a value
the call will not write (an imaginary part longer than the real one) still is
zero."""
import numpy as np
import pytest


@pytest.mark.parametrize("shape,n", [((6,), 6), ((2, 3), 6), ((6,), 4), ((2, 4), 5), ((3,), 0)])
def test_values_past_the_result_are_zero(pkg, shape, n):
    like = np.full(shape, 7.0)
    a = pkg._out(like, n)
    assert a.shape == shape and a.dtype == like.dtype and a is not like
    assert not a.reshape(-1)[n:].any()


def test_a_batch_sets_plane_threads_on_its_contexts(pkg, monkeypatch):
    """The call takes a context: a batch handed its own handle in a context's place."""
    handles = []

    class Lib:
        @staticmethod
        def sdft_ctx_set_plane_threads(handle, nt):
            handles.append((handle, nt))
            return 0

    monkeypatch.setattr(pkg, "lib", Lib)
    ctxs = [pkg.Context.__new__(pkg.Context) for _ in range(2)]
    for k, c in enumerate(ctxs):
        c._p = 100 + k
    b = pkg.Batch.__new__(pkg.Batch)
    b._ctxs, b._p = ctxs, 7
    b.set_plane_threads(128)
    for x in ctxs + [b]:
        x._p = None  # nothing to destroy
    assert handles == [(100, 128), (101, 128)]
