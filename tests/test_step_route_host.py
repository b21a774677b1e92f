"""CPU test: the calls that NewtonBonds.step hands to the float64 step driver, and those it
leaves to the Python control path, which refuses what it always refused."""
from types import SimpleNamespace

import numpy as np
import pytest


@pytest.mark.parametrize('max_iterations,native', [(12, True), (0, True), (31, True), (np.int64(12), True),
                                                   (32, False), (-1, False), (2.5, False), (12., False)])
def test_iteration_counts(max_iterations, native):
    import dpf_gb300
    solver = object.__new__(dpf_gb300.NewtonBonds)
    solver.profile, solver._graph = None, SimpleNamespace(n_sites=3)
    assert solver._native64_ready('fgmres', 'elastic', max_iterations) is native


@pytest.mark.parametrize('tolerances,native', [((1e-6, 2e-6), True), ((0, np.inf), True), ((np.float32(1e-6), np.nan), True),
                                               (('1e-6', 2e-6), False), ((1e-6, None), False)])
def test_tolerances(tolerances, native):
    import dpf_gb300
    solver = object.__new__(dpf_gb300.NewtonBonds)
    solver.profile, solver._graph = None, SimpleNamespace(n_sites=3)
    assert solver._native64_ready('fgmres', 'elastic', 12, 1e-6, tolerances) is native
    assert solver._native64_ready('fgmres', 'elastic', 12, None) is False
    assert solver._native64_ready('fgmres', 'elastic', 12, '1e-6') is False
