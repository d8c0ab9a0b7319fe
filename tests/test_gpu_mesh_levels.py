"""Mesh refinement level by level on the GPU, where counts are not read back between
levels: one leaf, more levels than are launched at a time, and more cells than the
first tables hold.  Integer decisions and FP64 rounding in a fixed order: equal to
the oracle bit for bit."""
import importlib

import numpy as np
import pytest

from oracle import mesh_oracle as MO

pytestmark = pytest.mark.gpu

CASES = {   # XL, base side, atoms, order, h, H, r, level, min_depth
    "one leaf": (1.0, 2.0, [[9.0, 0.0, 0.0]], 1, 0.5, 4.0, 0.1, -2.0, 0),
    "no atoms": (2.0, 1.0, np.zeros((0, 3)), 1, 0.5, 0.9, 0.1, -2.0, 0),
    "14 levels": (8.0, 16.0, [[0.7, -0.3, 0.2]], 1, 0.002, 20.0, 0.004, -3.0, 0),
    "110,592 cells": (3.0, 2.0, [[0.0, 0.0, 0.0]], 1, 50.0, 60.0, 0.5, 0.0, 4),
    "23 atoms": (4.0, 2.0, np.random.default_rng(3).uniform(-3, 3, (23, 3)), 2, 0.4, 2.0, 0.6, -2.0, 0),
}


@pytest.mark.parametrize("name", CASES)
def test_levels_match_oracle(native, pkg, name):
    M = importlib.import_module(pkg.__name__ + ".mesh")
    XL, side, atoms, order, h, H, r, level, min_depth = CASES[name]
    base = M.base_cells(XL, XL, XL, side)
    cells, ppc_c, ppc_f, nfine = M.refine_cells(base, atoms, order, h, H, r, level, min_depth)
    tab = MO.cell_table(MO.refine(MO.base_cells(XL, XL, XL, side), np.asarray(atoms, float), h, H, r, level, min_depth),
                        order)
    for k, v in zip(("cx", "cy", "cz", "dx", "dy", "dz", "ppc_c", "ppc_f"), (*cells, ppc_c, ppc_f)):
        assert np.array_equal(v.cpu().numpy(), tab[k]), k
    assert nfine == int(np.sum(tab["ppc_f"], dtype=np.int64))
