"""The energy law's passes against the oracle on graphs that straddle their
blocks and lanes, through the site records and without them, with moderate
multipliers and with multipliers whose exponentials overflow one by one but not
in a bond's sum.  Tolerances are those of the energy law's golden tests."""
import ctypes

import numpy as np
import pytest

from tests.helpers import host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,m', [(2, 1), (17, 33), (65, 129), (300, 2049)])
@pytest.mark.parametrize('far', [False, True])
def test_energy_forces_torques(n, m, far):
    import torch
    import dpf_gb300
    from dpf_gb300 import _lib
    from oracle import dem
    rng = np.random.default_rng(n)
    points = rng.normal(size=(n, 3))*2
    i = rng.integers(0, n, m)
    pairs = np.stack((i, (i + rng.integers(1, n, m)) % n), 1)
    if far:      # bonds between an even and an odd site only, whose multipliers cancel
        even = rng.integers(0, (n + 1)//2, m)*2
        pairs = np.stack((even, rng.integers(0, n//2, m)*2 + 1), 1)
    g = dict(points=points, radii=np.full(n, .3), pairs=pairs, areas=rng.uniform(.5, 1., m),
             contacts=points[pairs].mean(1) + .1*rng.normal(size=(m, 3)), masses=np.ones(n), fixed=np.zeros(n, bool))
    law = dpf_gb300.EnergyFoam(g, volume=False, young=1200., shear=480.)
    ref = dem.EnergyBonds(g['points'], g['radii'], pairs, g['areas'], g['contacts'], g['masses'], g['fixed'])
    theta = rng.normal(size=(n, 5))*.3 + (1450.*(-1.)**np.arange(n)[:, None] if far else 0.)
    x, q = points + .1*rng.normal(size=(n, 3)), rng.normal(size=(n, 4))*.2 + [1., 0, 0, 0]
    q /= np.linalg.norm(q, axis=1)[:, None]
    force, torque = ref.forces(theta, x, q)
    energy = ref.energy(theta, x, q)

    def check(f, tau, e):
        assert np.abs(host(f) - force).max() <= 1e-11*np.abs(force).max()
        assert np.abs(host(tau) - torque).max() <= 1e-11*np.abs(torque).max()
        assert abs(float(e) - energy) <= 1e-12*abs(energy)
    check(*law.forces(theta, x, q), law.energy(theta, x, q))
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=law.device)
    th, xd, qd = t(theta), t(x), t(q)
    f, tau, e = torch.empty_like(xd), torch.empty_like(xd), torch.empty(1, dtype=torch.float64, device=law.device)
    b = law._bonds
    _lib.call('dpf_bond_energy', ctypes.byref(b._graph), law.base.data_ptr(), th.data_ptr(), 5, xd.data_ptr(),
              qd.data_ptr(), law.n0.data_ptr(), law.ri.data_ptr(), law.rj.data_ptr(), f.data_ptr(), tau.data_ptr(),
              e.data_ptr(), law._wrench.data_ptr(), law._partials.data_ptr(), b._stream())
    check(f, tau, e)
