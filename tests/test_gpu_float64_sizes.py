"""The float64 passes, the two float64 PCGs and the reductions at the sizes where their
launches change shape, against the oracle: one lane a site for the blocks (from 12,288
sites), 256-thread reductions (from 19,456 sites), two 256-thread blocks an SM for the
PCGs (over 77,824 bonds), and reductions whose blocks take several rounds, the last with
idle lanes (over 131,072 sites).  Tolerances are the reference's bars, as in
test_gpu_float64_passes.py; sums of squares over 10^6 entries carry 1e-12 of themselves."""
import numpy as np
import pytest

from tests.helpers import host, rel
from tests.test_gpu_float64_passes import DT, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,m', [(12287, 40001), (12289, 77825), (20011, 90001), (131201, 262147)])
def test_trial_jacobian_blocks_and_norms(n, m):
    gpu, cpu, rng = _pair(n, m, contacts=True, seed=n)
    y, d, external = rng.normal(0, .02, (n, 6)), rng.normal(size=(n, 6)), rng.normal(size=(n, 6))
    want, got = cpu.trial(y), gpu.trial(gpu.tensor(y))
    for name in ('force', 'n', 'ri', 'rj', 'x', 'normal', 'fn', 'fs', 'mt', 'mb', 'offset'):
        assert rel(got[name], want[name]) < 1e-12, name
    assert rel(gpu.jacobian_vector(gpu.tensor(y), gpu.tensor(d), DT, None), cpu.jacobian_vector(y, d, DT, None)) < 2e-11
    gpu.prepare_scaling(got, DT)
    cpu.prepare_scaling(want, DT)
    for name in ('diagonal', 'block', 'units'):
        assert rel(getattr(gpu, name), getattr(cpu, name)) < 1e-12, name
    assert rel(gpu.preconditioner, cpu.preconditioner) < 1e-9
    assert rel(gpu.stiffness(gpu.tensor(d)), cpu.stiffness(d)) < 1e-12
    # the residual's norms [|r|, max |s|, |s|]: the pass that forms both, and the one that scales
    residual = cpu.residual(y, DT, external)
    scaled = cpu.scale_residual(residual)
    norms = [np.linalg.norm(residual), np.abs(scaled).max(), np.linalg.norm(scaled)]
    gpu._v = gpu._vec(gpu.v)
    out = gpu.tensor(np.full((n, 6), np.nan))
    assert rel(gpu._evaluate(gpu.tensor(y), DT, gpu.tensor(external), scaled=out), residual) < 1e-12
    got_norms, status = gpu._fetch(3, status=True)
    assert status == 0 and np.allclose(got_norms, norms, rtol=1e-9, atol=0) and abs(got_norms[0]/norms[0] - 1) < 1e-12
    assert rel(out, scaled) < 1e-9
    gpu._call('dpf_scale_residual', n, gpu.preconditioner.data_ptr(), gpu.units.data_ptr(),
              gpu.tensor(residual).data_ptr(), out.data_ptr(), gpu._scalars.data_ptr(), gpu._partials.data_ptr(),
              gpu._stream())
    again, _ = gpu._fetch(3)
    assert np.allclose(again, norms, rtol=1e-9, atol=0) and abs(again[0]/norms[0] - 1) < 1e-12
    assert rel(out, scaled) < 1e-9


@pytest.mark.parametrize('n,m', [(12289, 77825), (20011, 90001)])
def test_elastic_linear_and_balanced_solves(n, m):
    import dpf_gb300
    from oracle import dem
    gpu, cpu, rng = _pair(n, m, seed=n + 1)
    y, d = rng.normal(0, .02, (n, 6)), rng.normal(size=(n, 6))
    x, info = dpf_gb300.LinearBonds.solve_increment(gpu, gpu.tensor(d), DT)
    want, ref = dem.LinearBonds.solve_increment(cpu, d, DT)
    assert info['iterations'] == ref['iterations'] and rel(x, want) < 1e-7
    x, info = dpf_gb300.FiniteBonds.solve_increment(gpu, gpu.tensor(d), DT)
    want, ref = dem.FiniteBonds.solve_increment(cpu, d, DT)
    assert info['iterations'] == ref['iterations'] and rel(x, want) < 1e-6
    gpu.prepare_scaling(gpu.trial(gpu.tensor(y)), DT)
    cpu.prepare_scaling(cpu.trial(y), DT)
    cpu.inner_iterations = gpu.inner_iterations = 0
    assert rel(gpu.elastic_precondition(gpu.tensor(d), DT), cpu.elastic_precondition(d, DT)) < 1e-8
    assert gpu.inner_iterations == cpu.inner_iterations


@pytest.mark.parametrize('n,m', [(20011, 90001), (131201, 262147)])
def test_start_of_a_driven_step(n, m):
    """The first entry of a step's trace: the residual at rest over the step's scale, and the largest scaled one."""
    gpu, cpu, rng = _pair(n, m, seed=n + 2)
    dt, external = 1e-3, rng.normal(size=(n, 6))
    assert gpu._native64_ready('fgmres', 'elastic')
    _, info = gpu.step(dt, gpu.tensor(external), tolerance=1e-3, pose_tolerance=1.)
    y = np.zeros((n, 6))
    cpu.prepare_scaling(cpu.trial(y), dt)
    residual = cpu.residual(y, dt, external)
    free = ~cpu.fixed[:, None]
    scale = max(np.linalg.norm(dt*cpu.mass*cpu.v + .5*dt*dt*external), .5*dt*dt*np.linalg.norm(cpu.loads()*free), 1e-30)
    relative, local = info['residual_trace'][0]
    assert abs(relative/(np.linalg.norm(residual)/scale) - 1) < 1e-12
    assert abs(local/np.abs(cpu.scale_residual(residual)).max() - 1) < 1e-9
