"""The packed term rows equal the field-by-field ones for every kind of row
that was accepted (CPU)."""
import ctypes

import numpy as np
import pytest

import g2s_b200 as g


def by_field(terms):
    return (g.QskTerm * max(len(terms), 1))(*[g.QskTerm(int(t[0]), int(t[1]), int(t[2]), float(t[3]), float(t[4]))
                                              for t in terms])


ROWS = {
    "none": [],
    "tuples": [(0, 1, 2, -1.0, 0.25), (3, 0, 1, 1e-30, -0.0)],
    "lists": [[0, 1, 2, 0.1, 1 / 3], [5, 0, 0, 3, 4]],
    "numpy scalars": [(np.int64(4), np.int32(1), np.uint8(2), np.float32(0.1), np.float64(1 / 3))],
    "numpy rows": list(np.array([[0.0, 1.0, 2.0, 0.5, 0.25], [7.0, 0.0, 1.0, -3.0, 2.0]])),
    "floats for indices": [(1.0, 0.0, 2.0, 0.5, 0.5)],
    "longer rows": [(1, 0, 2, 0.5, 0.5, "x")],
    "beyond float32": [(1, 0, 2, 1e300, float("nan")), (1, 0, 2, float("inf"), -1e300)],
}


@pytest.mark.parametrize("rows", list(ROWS.values()), ids=list(ROWS))
def test_packed_terms(rows):
    a, b = g._terms(rows), by_field(rows)
    assert type(a) is type(b) and bytes(a) == bytes(b)


def test_rows_that_were_refused():
    for rows in ([(1, 2, 3)], [(None, 0, 0, 0.0, 0.0)], [("a", 0, 0, 0.0, 0.0)]):
        with pytest.raises((TypeError, ValueError, IndexError)):
            by_field(rows)
        with pytest.raises((TypeError, ValueError, IndexError)):
            g._terms(rows)
    assert ctypes.sizeof(g.QskTerm) == 20


@pytest.mark.parametrize("row", [
    {0: 3, 1: 1, 2: 2, 3: 0.5, 4: -0.25},                       # fields by key, not the keys
    np.array([3, 1, 2, 4, 5]),
    np.array([(3, 1, 2, 0.5, -0.25)], "i4,i4,i4,f4,f4")[0],
], ids=["mapping", "integer array", "record"])
def test_rows_by_index(row):
    rows = [(0, 1, 2, -1.0, 0.25), row]
    assert bytes(g._terms(rows)) == bytes(by_field(rows))
    assert bytes(g._terms([row])) == bytes(by_field([row]))


@pytest.mark.parametrize("make", [lambda: {3, 1, 2, 0, 4}, lambda: iter((0, 1, 2, 3, 4)),
                                  lambda: (x for x in (0, 1, 2, 3, 4)), lambda: {0: 1, 1: 1, 2: 1, 3: 1, 5: 1}],
                         ids=["set", "iterator", "generator", "mapping without a field"])
def test_rows_without_an_index_are_refused(make):
    for f in (by_field, g._terms):
        with pytest.raises((TypeError, KeyError)):
            f([make()])
