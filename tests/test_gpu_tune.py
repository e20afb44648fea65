"""The tuner sets the plans that it times, and no others: kinds 0 and 1 are also the plans of FFT<Dim>."""

import ctypes as ct

import pytest

from azeban_b200 import _lib, tune

pytestmark = pytest.mark.gpu


def _table(prec, L):
    got = []
    for kind in range(6):
        v = ct.c_int()
        _lib.check(_lib.lib.az_tune_get(prec, L, kind, ct.byref(v)))
        got.append(v.value)
    return got


@pytest.mark.parametrize("dim,N,M,tuned", [(2, 16, 24, ()), (3, 16, 24, (2,)), (3, 32, 384, (0, 2))])
@pytest.mark.parametrize("prec", [0, 1])
def test_autotune_sets_what_it_times(prec, dim, N, M, tuned):
    before = _table(prec, M)
    try:
        other = [1 - (v & 1) for v in before]
        for kind, v in enumerate(other):
            _lib.check(_lib.lib.az_tune_set(prec, M, kind, v))
        entries = tune.autotune(dim, N, "f64" if prec == 0 else "f32", M=M, reps=1)
        after = _table(prec, M)
        assert sorted(e["kind"] for e in entries) == list(tuned)
        for kind in range(6):
            if kind in tuned:
                assert after[kind] == next(e["variant"] for e in entries if e["kind"] == kind) in (0, 1)
            else:
                assert after[kind] == other[kind], kind
    finally:
        for kind, v in enumerate(before):
            _lib.check(_lib.lib.az_tune_set(prec, M, kind, v))
