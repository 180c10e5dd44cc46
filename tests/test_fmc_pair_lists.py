"""Monitor rows and weights of transmitter-receiver pairs (fmc._pair_lists)
for every way of naming steps and receivers, against a look-up per pair."""
import numpy as np
import pytest

from bfe_gb300.fmc import _pair_lists
from bfe_gb300.solver import SolverError

NDS = [np.array([3, 4, 5]), np.array([7]), np.array([9, 11])]
MON = [np.array([3, 4, 5, 7, 9, 11]), np.array([11, 9, 7, 5, 4, 3]), np.array([3, 4, 5, 7, 9, 11])]
WTS = [None, np.array([2.0]), np.array([0.5, -1.0])]
TX, RX = [0, 0, 1, 2, 2, 1, 0], [2, 0, 1, 0, 2, 2, 0]


def _plain(tx, rx, mon, nds, wts):
    p, s, w = [0], [], []
    for a, b in zip(tx, rx):
        m = np.asarray(mon[a])
        sel = [k for k in range(m.size) if m[k] in nds[b]]
        s += sel
        w += [1.0] * len(sel) if wts is None or wts[b] is None else list(wts[b])
        p.append(len(s))
    return p, s, w


def _objects(x):
    o = np.empty(len(x), object)
    o[:] = x
    return o


FORMS = dict(
    lists=(list, lambda m: m),
    integers=(lambda x: np.array(x, np.uint8), lambda m: m),
    objects=(_objects, lambda m: m),
    generator=(lambda x: (k for k in x), lambda m: m),
    strings=(lambda x: ["e%d" % k for k in x], lambda m: {"e%d" % k: v for k, v in enumerate(m)}),
    floats=(lambda x: [0.5 + k for k in x], lambda m: {0.5 + k: v for k, v in enumerate(m)}),
    tuples=(lambda x: [(k, 1) for k in x], lambda m: {(k, 1): v for k, v in enumerate(m)}),
    ragged=(lambda x: [(1,) * (k + 1) for k in x], lambda m: {(1,) * (k + 1): v for k, v in enumerate(m)}),
    far_apart=(lambda x: [k * 3 * 10 ** 18 for k in x], lambda m: {k * 3 * 10 ** 18: v for k, v in enumerate(m)}),
)


@pytest.mark.parametrize("wts", [None, WTS])
@pytest.mark.parametrize("form", sorted(FORMS))
def test_every_form_of_names(form, wts):
    name, table = FORMS[form]
    named = None if wts is None else table(wts)
    got = _pair_lists(name(TX), name(RX), table(MON), table(NDS), named)
    for a, b, t in zip(got, _plain(TX, RX, MON, NDS, wts), (np.int64, np.int64, float)):
        assert a.dtype == t and a.tolist() == b


def test_ends_with_the_shorter_list_and_none_at_all():
    got = _pair_lists(TX[:3], RX, MON, NDS, None)
    assert [x.tolist() for x in got] == [list(x) for x in _plain(TX[:3], RX[:3], MON, NDS, None)]
    assert [x.tolist() for x in _pair_lists([], [], MON, NDS, None)] == [[0], [], []]


@pytest.mark.parametrize("form", ["lists", "strings"])
def test_weights_that_do_not_match_are_refused(form):
    name, table = FORMS[form]
    with pytest.raises(SolverError):
        _pair_lists(name(TX), name(RX), table(MON), table(NDS), table([None, np.ones(4), None]))
