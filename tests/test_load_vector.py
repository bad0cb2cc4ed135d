"""Solver.load_vector builds F from the rows (id, fx, fy, fz) of the last set_bc."""
import numpy as np
import pytest

from gmgs import Solver


class Rows(Solver):
    def __init__(self, rows):
        self._loads = np.array(rows, dtype=np.float64).reshape(-1, 4)

    def num_nodes(self, level=1):
        return 5

    def close(self):
        pass


def test_later_rows_win():
    F = Rows([[2, 1, 2, 3], [5, 4, 5, 6], [2, 7, 8, 9]]).load_vector()
    assert np.array_equal(F.reshape(5, 3), [[0, 0, 0], [7, 8, 9], [0, 0, 0], [0, 0, 0], [4, 5, 6]])
    assert np.array_equal(Rows([]).load_vector(), np.zeros(15))


@pytest.mark.parametrize("node", [0, -1, 6, 10 ** 12])
def test_ids_that_set_bc_refuses_are_refused(node):
    with pytest.raises(ValueError):
        Rows([[1, 1, 1, 1], [node, 1, 2, 3]]).load_vector()
