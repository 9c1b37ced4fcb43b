"""Tokens and slots as a caller may hand them to a step: any kind of whole number, in any kind of iterable."""
from fractions import Fraction

import numpy as np
import pytest
import torch

from janas_b200.engine import Engine
from janas_b200.engine.engine import StepError, _ints

VALUES = [7, 0, -3, 2 ** 31 - 1]


@pytest.mark.parametrize("kind", [int, float, str, np.int64, np.int32, np.float64, Fraction, torch.tensor])
@pytest.mark.parametrize("hold", [list, tuple, iter, lambda v: (x for x in v), lambda v: dict.fromkeys(v).keys()])
def test_packing(kind, hold):
    for values in (VALUES, VALUES + [11, 12, 13]):          # short lists are packed another way
        assert list(_ints(hold([kind(v) for v in values]))) == values


@pytest.mark.parametrize("values", [np.array(VALUES), np.array(VALUES, dtype=np.float64), torch.tensor(VALUES), range(5)])
def test_packing_of_arrays(values):
    assert list(_ints(values)) == [int(v) for v in values]


@pytest.mark.parametrize("n", [1, 4, 5, 40])
def test_packing_beyond_32_bits(n):
    assert list(_ints([2 ** 40 + 5] * n)) == [5] * n        # the low 32 bits, as a C int takes them


def test_packing_of_nothing_leaves_a_place():
    for none in ([], (), iter([]), np.array([], dtype=np.int32)):
        assert list(_ints(none)) == [0]


@pytest.mark.parametrize("tokens", [[], [5], (5,), iter([5]), iter([5.0]), np.array([5])])
def test_a_decode_step_wants_a_token_for_every_slot(tokens):
    eng = object.__new__(Engine)            # refused before the library is called
    with pytest.raises(StepError, match="tokens for 2 sequences"):
        eng.decode_begin([0, 1], tokens)


@pytest.mark.parametrize("kind", [list, tuple, np.array, torch.tensor])
def test_packing_of_a_step(kind):
    """All entries' tokens and wanted places go into one array: every piece has its own, whatever holds them."""
    import ctypes
    from janas_b200.engine.engine import StepEntry
    entries = [(3, kind([5, 6, 7]), [0, 2]), StepEntry(9, kind([2 ** 31 - 1]), ()), (4, kind([8, 1]), kind([1])), (0, [], []),
               (2, [4.0, Fraction(3)], [1])]
    pieces, keep, wanted = object.__new__(Engine)._pieces(entries)
    assert wanted == 4 and len(pieces) == 5

    def at(address, n):
        return [ctypes.c_int32.from_address(address + 4 * i).value for i in range(n)]

    got = [(p.slot, at(p.tokens, p.n), at(p.want, p.n_want)) for p in pieces]
    assert got == [(3, [5, 6, 7], [0, 2]), (9, [2 ** 31 - 1], []), (4, [8, 1], [1]), (0, [], []), (2, [4, 3], [1])]
    assert all(p.tokens and p.want for p in pieces)
