"""The float64 step driver against the Python control path: the same iteration
counts and decisions, states to rounding (both solve the same float64 systems;
sums are taken in another order), for both preconditionings, a restarted FGMRES,
ragged sizes, given contacts and the failure outcomes.

Positions, velocities and rotations agree to 1e-10 relative.  A bond force is its
stiffness times the difference of two increments, so it carries their rounding:
64 units in the last place of k |y| beside 1e-10 of itself."""
import numpy as np
import pytest

from tests.helpers import host, rel

pytestmark = pytest.mark.gpu

STATE = ('x', 'v', 'rotation', 'normal', 'offset', 'fn', 'fs', 'mt', 'mb')


def _pair(m, seed=1, contacts=False, young=1e5):
    import dpf_gb300
    foam = dpf_gb300.jittered_lattice_foam(m, seed=seed, young=young)
    args = [foam[k] for k in ('points', 'radii', 'pairs', 'areas', 'masses', 'fixed')]
    given = None
    if contacts:
        p = foam['points'][foam['pairs']]
        given = p.mean(1) + .02*foam['h']*np.random.default_rng(seed).normal(size=(len(p), 3))
    solvers = [dpf_gb300.NewtonBonds(*args, contacts=given, young=foam['young'], shear=foam['shear'])
               for _ in range(2)]
    solvers[0].native = False
    assert solvers[1]._native64_ready('fgmres', 'elastic', 12)
    return dpf_gb300.gravity_load(foam), *solvers


def _same(python, native, travel):
    """travel: the largest increment so far."""
    rounding = dict(fn='kn', fs='ks', mt='kt', mb='kb')
    for name in STATE:
        a, b = host(getattr(native, name)), host(getattr(python, name))
        floor = 64*2.**-53*np.linalg.norm(host(getattr(python, rounding[name])))*travel if name in rounding else 0.
        assert np.linalg.norm(a - b) <= 1e-10*np.linalg.norm(b) + floor, name
    for name in ('n', 'ri', 'rj', 'diagonal', 'block', 'preconditioner', 'units'):
        assert rel(getattr(native, name), getattr(python, name)) < 1e-9, name
    assert native.time == python.time and native.inner_iterations == python.inner_iterations


@pytest.mark.parametrize('m,contacts,preconditioning', [(2, False, 'elastic'), (5, True, 'elastic'), (7, False, 'block'),
                                                        (12, True, 'elastic')])
def test_steps_match_the_python_path(m, contacts, preconditioning):
    load, python, native = _pair(m, contacts=contacts)
    travel = 0.
    for _ in range(3):
        wp, ip = python.step(2e-3, python.tensor(load), preconditioning=preconditioning)
        wn, inn = native.step(2e-3, native.tensor(load), preconditioning=preconditioning)
        for key in ('nonlinear_iterations', 'krylov_iterations', 'cg_iterations'):
            assert ip[key] == inn[key], key
        assert abs(wp - wn) <= 1e-10*abs(wp)
        assert np.allclose(ip['residual_trace'], inn['residual_trace'], rtol=1e-3, atol=1e-12)
        assert abs(ip['max_step_rotation'] - inn['max_step_rotation']) <= 1e-10*ip['max_step_rotation']
        travel += float(2e-3*python.v.abs().max())
        _same(python, native, travel)


@pytest.mark.parametrize('factor', [1., 1.03])
@pytest.mark.parametrize('linear', [True, False])
def test_prestressed_steps_with_and_without_the_stored_linearisation(factor, linear):
    """A random history, committed normals that are unit vectors and not (the stored
    linearisation does not hold for those), and the products formed anew."""
    load, python, native = _pair(5, contacts=True)
    rng = np.random.default_rng(4)
    m = python.n_bonds
    h = {name: rng.normal(size=(m, 3))*1e-2 for name in ('fs', 'mb')}
    h.update({name: rng.normal(size=m)*1e-2 for name in ('fn', 'mt')}, normal=host(python.normal)*factor)
    for s in (python, native):
        for name, value in h.items():
            setattr(s, name, s.tensor(value))
    if not linear:
        native._native64_buffers()
        native._native64_linear = None
        native._native64_desc = None
    _, ip = python.step(1e-3, python.tensor(load))
    _, inn = native.step(1e-3, native.tensor(load))
    for key in ('nonlinear_iterations', 'krylov_iterations', 'cg_iterations'):
        assert ip[key] == inn[key], key
    _same(python, native, float(1e-3*python.v.abs().max()))


def test_restarted_krylov_cycles():
    """A stiff step without the elastic preconditioner needs more than one cycle of 32."""
    load, python, native = _pair(6, young=3e7)
    _, ip = python.step(5e-3, python.tensor(load), preconditioning='block')
    _, inn = native.step(5e-3, native.tensor(load), preconditioning='block')
    assert ip['krylov_iterations'] > 32
    assert abs(ip['krylov_iterations'] - inn['krylov_iterations']) <= 1
    assert rel(native.x, python.x) < 1e-8 and rel(native.v, python.v) < 1e-5


def test_outcomes_and_untouched_state():
    from dpf_gb300 import SubdivideError
    load, python, native = _pair(5)
    twist = np.zeros_like(load)
    twist[:, 3:] = np.random.default_rng(2).normal(size=(len(load), 3))*1e4      # turns far beyond the guard
    for force, kw, word in ((twist, {}, None), (load, dict(max_iterations=0), 'did not converge')):
        messages = []
        for s in (python, native):
            before = {name: host(getattr(s, name)).copy() for name in STATE}
            with pytest.raises(SubdivideError) as error:
                s.step(1e-3, s.tensor(force), **kw)
            messages.append(str(error.value).split('(')[0])
            assert all(np.array_equal(host(getattr(s, name)), before[name]) for name in STATE)
        assert messages[0] == messages[1]
        assert word is None or word in messages[0]
    _, info = native.step(1e-3, native.tensor(load))
    assert info['nonlinear_iterations'] >= 1


def test_replaced_methods_keep_the_python_path():
    _, python, native = _pair(3)
    assert not python._native64_ready('fgmres', 'elastic', 12)
    assert not native._native64_ready('dense', 'elastic')
    assert not native._native64_ready('fgmres', 'elastic', linear_tolerance=1e-15)
    calls = []
    plain = native.jacobian_vector
    native.jacobian_vector = lambda *a: calls.append(1) or plain(*a)
    load = np.zeros((27, 6))
    load[-1, 2] = -1.
    native.step(1e-3, native.tensor(load))
    assert calls


@pytest.mark.parametrize('iterations', [1, 2, 3])
@pytest.mark.parametrize('preconditioning', ['elastic', 'block'])
def test_rejected_full_steps(iterations, preconditioning):
    """A pull whose first Newton corrections are halved: the iterate's tangent, blocks and inverses are
    there again for the shorter candidates.  The step is cut off after a few iterations and its message
    carries the residual and the pose defect of the last iterate in six digits (one unit of the last)."""
    import dpf_gb300
    load, python, native = _pair(3)
    load[:, :3] += np.random.default_rng(1).normal(size=(len(load), 3))*100*np.abs(load).max()
    values = []
    for s in (python, native):
        with pytest.raises(dpf_gb300.SubdivideError, match='did not converge') as error:
            s.step(1e-2, s.tensor(load), max_iterations=iterations, preconditioning=preconditioning)
        values.append([float(v) for v in str(error.value).split('(')[1].rstrip(')').split(',')])
    assert np.allclose(values[0], values[1], rtol=2e-5, atol=0), values
