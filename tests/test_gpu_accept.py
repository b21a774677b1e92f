"""A step committed again from its increment gives the bits of the first time: the accept
kernel behind ``dpf_accept_step`` (which an adjoint's replay runs) against the float64 step
driver's and the mixed one's, at velocities and increments whose 2 y / dt and v nearly cancel
(where a product that is rounded before the difference would show)."""
import numpy as np
import pytest

from tests.test_gpu_driver import pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('m', [3, 9])
@pytest.mark.parametrize('mixed', [False, True])
def test_recommitted_velocity_and_rotation(m, mixed):
    import dpf_gb300
    from dpf_gb300 import _lib
    foam = dpf_gb300.jittered_lattice_foam(m, seed=m)
    args = (foam['points'], foam['radii'], foam['pairs'], foam['areas'], foam['masses'], foam['fixed'])
    kw = dict(young=foam['young'], shear=foam['shear'])
    if mixed:
        _, _, s = pair(m=m, seed=m)
    else:
        s = dpf_gb300.NewtonBonds(*args, **kw)
    seen = []
    s._accepted = lambda y: seen.append(y.clone())
    load, dt = dpf_gb300.gravity_load(foam)*4., 2e-3
    s.step(dt, s.tensor(load), tolerance=1e-6)
    # a drift of all bodies: v = 2 y / dt - v up to the step's small changes
    s.v = s.v + s.tensor(np.where(foam['fixed'][:, None], 0., .05*np.sin(np.arange(6*len(foam['points'])).reshape(-1, 6))))
    v, rotation = s.v.clone(), s.rotation.clone()
    s.step(dt, s.tensor(load), tolerance=1e-6)
    # the mixed driver's increment is one of the two vectors it swaps
    y = min(s._native_vectors[:2], key=lambda t: float((2/dt*t - v - s.v).abs().max())) if mixed else seen[-1]
    _lib.call('dpf_accept_step', s.n_sites, y.data_ptr(), dt, v.data_ptr(), rotation.data_ptr(), s._stream())
    assert np.array_equal(v.cpu().numpy(), s.v.cpu().numpy())
    assert np.array_equal(rotation.cpu().numpy(), s.rotation.cpu().numpy())
