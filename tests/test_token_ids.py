"""Token lists of a step: what goes through ``array`` and what it refuses give what numpy alone would."""
import numpy as np
import pytest

from quicknn_b200.engine.engine import token_ids


@pytest.mark.parametrize("tokens", [[1, 2, 3], [0], [], [True, False], [-5, 2 ** 62], [np.int32(4), np.uint8(7)], [1.7, 2.0], ["3"], [[1, 2], [3, 4]],
                                    (1, 2), range(3), np.array([[1, 2]], np.int32), np.array([3.5])], ids=str)
def test_the_numbers_of_numpy_alone(tokens):
    want = np.asarray(tokens, dtype=np.int64).reshape(-1)
    got = token_ids(tokens)
    assert got.dtype == np.int64 and got.shape == want.shape and (got == want).all()


@pytest.mark.parametrize("tokens", [[2 ** 63], [-2 ** 63 - 1], [None], [1, "a"], [[1], [2, 3]]], ids=str)
def test_the_refusals_of_numpy_alone(tokens):
    with pytest.raises(Exception) as want:
        np.asarray(tokens, dtype=np.int64).reshape(-1)
    with pytest.raises(want.type):
        token_ids(tokens)


def test_a_list_that_changes_later_does_not_change_what_was_taken():
    tokens = [1, 2, 3]
    got = token_ids(tokens)
    tokens[0] = 9
    assert got.tolist() == [1, 2, 3]
