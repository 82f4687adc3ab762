"""The finals of SALI, MEGNO and FLI read their states by field name and hand out sums of their own: other layouts of the
same fields give the same columns, and writing to a column leaves the states alone."""
from __future__ import annotations

import numpy as np
import pytest

from chaos_b200 import FLI, MEGNO, SALI

REDUCERS = [SALI(), MEGNO(), FLI()]


def _states(r, n=17):
    rng = np.random.default_rng(3)
    st = np.zeros(n, dtype=r.dtype(2, 2))
    for name in st.dtype.names:
        if st.dtype[name] == "<f8":
            st[name] = rng.normal(size=n)
        elif name in ("n", "K"):
            st[name] = rng.integers(0, 50, n) if name == "K" else 50
    return st


def _same(a, b):
    assert a.keys() == b.keys()
    for key in a:
        assert np.array_equal(a[key], b[key]), key


def _relaid(st, kind):
    names = [nm for nm in st.dtype.names if not nm.startswith("_")]
    if kind == "columns":
        return {nm: st[nm].copy() for nm in names}
    dt = {"reversed": [(nm, st.dtype[nm]) for nm in reversed(names)],
          "padded": [f for i, nm in enumerate(names) for f in ((f"_gap{i}", "V8"), (nm, st.dtype[nm]))],
          "big endian": [(nm, st.dtype[nm].newbyteorder(">")) for nm in names]}[kind]
    out = np.zeros(len(st), dtype=dt)
    for nm in names:
        out[nm] = st[nm]
    return out


@pytest.mark.parametrize("kind", ["reversed", "padded", "big endian", "columns"])
@pytest.mark.parametrize("r", REDUCERS, ids=repr)
def test_other_layouts_give_the_same_columns(r, kind):
    st = _states(r)
    _same(r.finals(_relaid(st, kind)), r.finals(st))


@pytest.mark.parametrize("r", REDUCERS, ids=repr)
def test_strided_states(r):
    st = _states(r)
    _same(r.finals(st[::2]), r.finals(st[::2].copy()))
    _same(r.finals(st[:0]), {key: v[:0] for key, v in r.finals(st).items()})


@pytest.mark.parametrize("r", REDUCERS, ids=repr)
def test_sums_are_arrays_of_their_own(r):
    st = _states(r)
    before, fin = st.copy(), r.finals(st)
    for key in ("sum", "comp"):
        assert fin[key].flags.owndata and fin[key].flags.c_contiguous
        fin[key][:] = -1.0
    assert st.tobytes() == before.tobytes()
