"""Restarts of the mixed-precision FGMRES: a chain so stiff for its step that 80
iterations of the elastic PCG precondition it poorly, and a solve takes more than one
cycle of 32 Arnoldi steps.  The step converges (its residual is formed again by the
float64 solver), on the Python control path and, bit for bit, through the driver."""
import numpy as np
import pytest

from tests.test_gpu_driver import assert_same_info, assert_same_state

pytestmark = pytest.mark.gpu

DT, TOLERANCE = .1, 1e-3      # the floor of the float32 passes: a few 1e-4 of the loads on such a chain


def _chain(cls, n, young=1e8):
    points = np.stack((np.arange(n), np.zeros(n), np.zeros(n)), 1).astype(float)
    pairs = np.stack((np.arange(n - 1), np.arange(1, n)), 1)
    s = cls(points, np.full(n, .5), pairs, np.ones(n - 1), np.ones(n), np.arange(n) == 0, young=young, shear=.4*young)
    load = np.zeros((n, 6))
    load[-1, 0], load[-1, 2] = 1e-6*young, 1e-9*young
    return s, s.tensor(load)


@pytest.mark.parametrize('n', [300, 1000])
def test_restarted_cycles_converge(n):
    import dpf_gb300
    (python, load), (native, _) = (_chain(dpf_gb300.MixedNewtonBonds, n) for _ in range(2))
    exact, _ = _chain(dpf_gb300.NewtonBonds, n)
    python.native = False
    for s in (python, native):
        s._end_variant = 0
    for step in range(2):      # the first step of a solver runs on the Python path
        start = {k: getattr(python, k).clone() for k in ('x', 'v', 'rotation', 'normal', 'offset', 'fn', 'fs', 'mt', 'mb')}
        work, info = python.step(DT, load, tolerance=TOLERANCE, linear_tolerance=1e-5)
        assert native._native_ready('fgmres', 'elastic') == (step > 0)
        work_native, info_native = native.step(DT, load, tolerance=TOLERANCE, linear_tolerance=1e-5)
        assert info['krylov_iterations'] > 32*info['nonlinear_iterations'] > 0
        assert work == work_native
        assert_same_info(info, info_native)
        assert_same_state(python, native)
        for name, value in start.items():
            setattr(exact, name, value)
        residual = exact.residual(.5*DT*(python.v + start['v']), DT, load)
        free = ~exact.fixed[:, None]
        scale = max(float((exact.mass*start['v']*DT + .5*DT*DT*load).norm()), .5*DT*DT*float((exact.loads()*free).norm()))
        # the increment read back from the velocity carries a rounding of 2^-52 of both, times the stiffness
        rounding = DT*DT*float(exact.kn.max())*2.**-50*float((DT*python.v).norm())
        assert float((residual*free).norm()) <= 1.01*TOLERANCE*scale + rounding
