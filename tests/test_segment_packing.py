"""dslash_segments takes what the fields of QcuHopSegment take, and refuses what they refuse (no GPU: the
library call is a stand-in that keeps the list)."""
import ctypes

import pytest

import mrhs_qcu_gb300 as Q

PLAIN = dict(lattice=(4, 4, 6, 8), gauge=0x1000, gauge_two_row=0x2000, in_=0x3000, out=0x4000, x=0x5000, a=-0.5, b=2,
             nrhs=12, parity=1, dagger=1, antiperiodic_t=True)


class _Library:
    def qcuDslashSegments(self, arr, n, n_colors, precision, stream):
        self.seen = [bytes(arr[i]) for i in range(n)]
        return 0


@pytest.fixture
def pack(monkeypatch):
    library = _Library()
    monkeypatch.setattr(Q, "lib", lambda: library)

    def call(segments):
        Q.dslash_segments(segments, 3, 1)
        return library.seen

    return call


def _by_fields(d):
    g = Q.QcuHopSegment()
    g.lattice = (ctypes.c_int * 4)(*d["lattice"])
    for k in ("gauge", "gauge_two_row", "in_", "out", "x", "a", "b", "nrhs", "parity", "dagger", "antiperiodic_t"):
        setattr(g, k, d[k])
    return bytes(g)


@pytest.mark.parametrize("change", [
    {}, {"gauge": ctypes.c_void_p(0x1000)}, {"x": None}, {"x": ctypes.c_void_p(None)},
    {"in_": ctypes.c_void_p(0x3000), "out": ctypes.c_void_p(0x4000)}, {"nrhs": ctypes.c_int(12)}, {"lattice": (4, 4, 6)},
    {"a": ctypes.c_double(0.25)}, {"parity": True}, {"nrhs": 2 ** 31}, {"gauge": 2 ** 64 - 16},
])
def test_takes_what_the_fields_take(pack, change):
    d = dict(PLAIN, **change)
    assert pack([PLAIN, d]) == [_by_fields(PLAIN), _by_fields(d)]
    assert pack([]) == []


@pytest.mark.parametrize("change,error", [
    ({"nrhs": 1.5}, TypeError), ({"in_": "field"}, TypeError), ({"a": None}, TypeError), ({"nrhs": None}, TypeError),
    ({"lattice": (4, 4, 4, 4, 4)}, IndexError),
])
def test_refuses_what_the_fields_refuse(pack, change, error):
    with pytest.raises(error):
        pack([dict(PLAIN, **change)])
