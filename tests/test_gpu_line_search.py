"""Newton steps whose first full corrections are rejected and whose shorter ones lead to
convergence: chains held at both ends and loaded across.  Their shear is soft, their
stretching stiff, so the linear model overshoots (by the merit, or beyond the guard on the
normals).  Behind a rejected full step the drivers restore the iterate's tangent, blocks,
inverses and linearisation: the float64 driver against the Python control path, the
mixed one bit for bit.

Tolerances: the linear solves and the residual go to 1e-10, so two float64 paths differ by
1e-10 of the loads in their residuals.  The softest motion that the loads drive has a
stiffness of shear/young = 1e-3 of the stiffest: 1e-7 in the increment."""
import numpy as np
import pytest

from tests.helpers import host, rel
from tests.test_gpu_driver import assert_same_info, assert_same_state

pytestmark = pytest.mark.gpu

DT = .5
CASES = [(3, 1e-2, .8), (3, 1e-3, 3.), (4, 1e-3, 1.5), (7, 1e-3, 1.5)]


def _chain(cls, n, shear, load):
    young = 1e4
    points = np.stack((np.arange(n), .01*np.random.default_rng(0).normal(size=n), np.zeros(n)), 1)
    pairs = np.stack((np.arange(n - 1), np.arange(1, n)), 1)
    fixed = np.zeros(n, bool)
    fixed[[0, -1]] = True
    s = cls(points, np.full(n, .5), pairs, np.ones(n - 1), np.ones(n), fixed, young=young, shear=shear*young)
    force = np.zeros((n, 6))
    force[1:-1, 2] = load*shear*young
    return s, s.tensor(force)


def _recording(base):
    """The solver on the Python control path, with the merit and guards of every candidate."""
    class Recording(base):
        def _line_merit(self, *args):
            out = super()._line_merit(*args)
            self.evaluations = getattr(self, 'evaluations', 0) + 1
            return out
    return Recording


@pytest.mark.parametrize('n,shear,load', CASES)
@pytest.mark.parametrize('preconditioning', ['elastic', 'block'])
@pytest.mark.parametrize('linear', [True, False])
def test_float64(n, shear, load, preconditioning, linear):
    import dpf_gb300
    python, force = _chain(_recording(dpf_gb300.NewtonBonds), n, shear, load)
    native, _ = _chain(dpf_gb300.NewtonBonds, n, shear, load)
    native._native64_linear = linear
    assert native._native64_ready('fgmres', preconditioning, 30, 1e-10) and not python._native64_ready('fgmres', preconditioning)
    kw = dict(tolerance=1e-10, linear_tolerance=1e-10, max_iterations=30, preconditioning=preconditioning)
    wp, ip = python.step(DT, force, **kw)
    wn, inn = native.step(DT, force, **kw)
    assert python.evaluations > ip['nonlinear_iterations']      # full steps were rejected
    assert ip['nonlinear_iterations'] == inn['nonlinear_iterations']
    assert abs(wp - wn) <= 1e-7*abs(wp)
    for name in ('x', 'v', 'rotation', 'normal', 'fn', 'fs', 'mb', 'n', 'ri', 'rj', 'diagonal', 'block', 'preconditioner'):
        assert rel(getattr(native, name), getattr(python, name)) < 1e-7, name
    # the iterates on the way: every entry of the trace above the last one's rounding
    a, b = np.array(ip['residual_trace']), np.array(inn['residual_trace'])
    assert np.abs(a - b).max() <= 1e-7*np.abs(a).max()


@pytest.mark.parametrize('n,shear,load', CASES)
def test_mixed(n, shear, load):
    import dpf_gb300
    python, force = _chain(_recording(dpf_gb300.MixedNewtonBonds), n, shear, load)
    native, _ = _chain(dpf_gb300.MixedNewtonBonds, n, shear, load)
    kw = dict(tolerance=1e-5, max_iterations=30)
    for s in (python, native):
        s._end_variant = 0
        s.step(1e-3, force*1e-3, **kw)      # sets up the sweep on the Python path
    python.evaluations = 0
    assert native._native_ready('fgmres', 'elastic') and not python._native_ready('fgmres', 'elastic')
    wp, ip = python.step(DT, force, **kw)
    wn, inn = native.step(DT, force, **kw)
    assert python.evaluations > ip['nonlinear_iterations']
    assert wp == wn
    assert_same_info(ip, inn)
    assert_same_state(python, native)
