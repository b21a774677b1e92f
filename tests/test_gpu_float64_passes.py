"""The float64 bond and site passes and the two float64 PCGs against the oracle
on graphs that straddle their warps, lanes and branches: site and bond counts
off the multiples of 32, sites without bonds, offsets zero and not, committed
normals that are unit vectors and not, spins on both sides of the small-angle
series.  Tolerances are the reference's bars (force and K q 1e-12, JVP 2e-11,
blocks 1e-12, inner CG 1e-8)."""
import numpy as np
import pytest

from tests.helpers import host, rel

pytestmark = pytest.mark.gpu

DT = 1e-2


def _pair(n, m, contacts=False, unit=True, seed=0):
    """The same random bonded sites in the CUDA solver and in the oracle, with a random history."""
    import dpf_gb300
    from oracle import dem
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n**(1/3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)]*3, indexing='ij'), -1).reshape(-1, 3)[:n]
    points = grid + rng.uniform(-.2, .2, (n, 3))
    pairs = np.zeros((0, 2), np.int64)
    if n > 1:
        i = rng.integers(0, n, m)
        pairs = np.stack((i, (i + rng.integers(1, n, m)) % n), 1)
    radii = rng.uniform(.3, .6, n)
    given = None
    if contacts:
        given = points[pairs].mean(1) + rng.normal(0, .1, (len(pairs), 3))
    args = (points, radii, pairs, rng.uniform(.5, 1., len(pairs)), rng.uniform(.5, 2., n), np.arange(n) % 5 == 3)
    gpu = dpf_gb300.NewtonBonds(*args, contacts=given)
    cpu = dem.NewtonBonds(*args, contacts=given)
    state = dict(fn=rng.normal(size=len(pairs)), mt=rng.normal(size=len(pairs)), fs=rng.normal(size=(len(pairs), 3)),
                 mb=rng.normal(size=(len(pairs), 3)), v=rng.normal(size=(n, 6)))
    state['normal'] = cpu.normal.copy()
    if not unit:
        state['normal'] = state['normal']*(1 + .1*rng.random((len(pairs), 1)))
    for name, value in state.items():
        setattr(cpu, name, value)
        setattr(gpu, name, gpu.tensor(value))
    return gpu, cpu, rng


@pytest.mark.parametrize('n,m', [(1, 0), (2, 1), (15, 31), (17, 33), (65, 255), (300, 2049)])
@pytest.mark.parametrize('contacts,unit', [(False, True), (True, True), (True, False)])
def test_trial_jacobian_and_blocks(n, m, contacts, unit):
    gpu, cpu, rng = _pair(n, m, contacts, unit, seed=n)
    y = rng.normal(0, .02, (n, 6))
    d = rng.normal(size=(n, 6))
    want, got = cpu.trial(y), gpu.trial(gpu.tensor(y))
    for name in ('force', 'n', 'ri', 'rj', 'x', 'normal', 'fn', 'fs', 'mt', 'mb', 'offset'):
        assert rel(got[name], want[name]) < 1e-12 or np.abs(host(got[name]) - want[name]).max() < 1e-14, name
    external = rng.normal(size=(n, 6))
    assert rel(gpu.residual(gpu.tensor(y), DT, gpu.tensor(external)), cpu.residual(y, DT, external)) < 1e-12
    assert rel(gpu.jacobian_vector(gpu.tensor(y), gpu.tensor(d), DT, None), cpu.jacobian_vector(y, d, DT, None)) < 2e-11
    # spins beyond the series and normals far turned (no guard on the product)
    y = rng.normal(0, [.1, .1, .1, 2., 2., 2.], (n, 6))
    assert rel(gpu.jacobian_vector(gpu.tensor(y), gpu.tensor(d), DT, None), cpu.jacobian_vector(y, d, DT, None)) < 2e-11
    gpu.prepare_scaling(got, DT)
    cpu.prepare_scaling(want, DT)
    for name in ('diagonal', 'block', 'units'):
        assert rel(getattr(gpu, name), getattr(cpu, name)) < 1e-12, name
    assert rel(gpu.preconditioner, cpu.preconditioner) < 1e-9
    assert rel(gpu.scale_residual(gpu.tensor(d)), cpu.scale_residual(d)) < 1e-9
    assert rel(gpu.stiffness(gpu.tensor(d)), cpu.stiffness(d)) < 1e-12 or m == 0
    cpu.inner_iterations = gpu.inner_iterations = 0
    assert rel(gpu.elastic_precondition(gpu.tensor(d), DT), cpu.elastic_precondition(d, DT)) < 1e-8
    assert gpu.inner_iterations == cpu.inner_iterations
    # down to rounding and some iterations past it
    exact = np.linalg.solve(_matrix(cpu, n), (cpu.block@(cpu.units*d)[:, :, None]*~cpu.fixed[:, None, None]).ravel()) \
        if n <= 65 else None
    if exact is not None:
        x = gpu.elastic_precondition(gpu.tensor(d), DT, tolerance=1e-14, max_iterations=400)
        assert rel(x, exact.reshape(n, 6)/cpu.units) < 1e-8


def _matrix(cpu, n):
    eye = np.eye(6*n)
    return np.stack([cpu._operator(column.reshape(n, 6), .25*DT*DT).ravel() for column in eye], 1)


@pytest.mark.parametrize('n,m', [(1, 0), (17, 33), (65, 255), (300, 2049)])
def test_linear_and_balanced_solves(n, m):
    import dpf_gb300
    gpu, cpu, rng = _pair(n, m, seed=n + 1)
    b = rng.normal(size=(n, 6))
    x, info = dpf_gb300.LinearBonds.solve_increment(gpu, gpu.tensor(b), DT)
    from oracle import dem
    want, ref = dem.LinearBonds.solve_increment(cpu, b, DT)
    assert info['iterations'] == ref['iterations']
    assert rel(x, want) < 1e-7
    x, info = dpf_gb300.FiniteBonds.solve_increment(gpu, gpu.tensor(b), DT)
    want, ref = dem.FiniteBonds.solve_increment(cpu, b, DT)
    assert info['iterations'] == ref['iterations']
    assert rel(x, want) < 1e-6
