"""A mesh with more cells than the first table holds is built in two calls: no error stays behind."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
mesh = importlib.import_module("treecode-accelerated-green-iteration_gb300.mesh")


def test_no_error_is_left_by_a_larger_mesh(native):
    native.lib().tagi_clear_error()
    base = np.array([[-4.0, 4.0, -4.0, 4.0, -4.0, 4.0]])
    cells, ppc_c, ppc_f, _ = mesh.refine_cells(base, np.zeros((0, 3)), 3, 1.0, 10.0, 1.0, 0.0, min_depth=5)
    assert len(cells[0]) == 8**5 > 16384 and len(ppc_c) == len(ppc_f) == 8**5
    assert native.last_error()[0] == 0
