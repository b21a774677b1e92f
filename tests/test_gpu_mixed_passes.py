"""The mixed-precision step driver's joined passes: bit-identical to the Python
control path at sizes off every block and warp edge, for lazy and eager commits,
committed and refreshed starts; and the packed bond-end records against their
definition (copies and single float32 products: exact)."""
import ctypes

import numpy as np
import pytest

from tests.helpers import host
from tests.test_gpu_driver import assert_same_info, assert_same_state, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('m', [2, 3, 7, 17])
@pytest.mark.parametrize('lazy', [False, True])
def test_driver_equals_python_path(m, lazy):
    import dpf_gb300
    foam, python, native = pair(m=m, seed=m, refresh=2)
    load = dpf_gb300.gravity_load(foam)*4.0
    for s in (python, native):
        s.lazy_history = lazy
    for step in range(5):
        out = [s.step(2e-3, s.tensor(load), tolerance=1e-6) for s in (python, native)]
        assert out[0][0] == out[1][0]
        assert_same_info(out[0][1], out[1][1])
        assert_same_state(python, native)


@pytest.mark.parametrize('n,m', [(2, 1), (17, 33), (129, 400)])
@pytest.mark.parametrize('sites', [False, True])
def test_packed_ends(n, m, sites):
    import torch
    from dpf_gb300 import _lib
    from tests.test_gpu_float64_passes import _pair
    gpu, cpu, rng = _pair(n, m, seed=n)
    lib, alpha = _lib.load(), .37
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a)).to(gpu.device)
    data = rng.normal(size=lib.dpf_mixed_bond_floats(m)).astype(np.float32)
    P = rng.normal(size=(n, 6, 6)).astype(np.float32)
    mass = rng.uniform(1, 2, (n, 6)).astype(np.float32)
    data_d, P_d, mass_d = dev(data), dev(P), dev(mass)
    ends, p24, site4 = (torch.full((k,), -7., dtype=torch.float32, device=gpu.device)
                        for k in (lib.dpf_end_floats(m), 24*n, 4*n))
    _lib.call('dpf_end_pack', ctypes.byref(gpu._graph), data_d.data_ptr(), alpha, P_d.data_ptr(), mass_d.data_ptr(),
              gpu.fixed.data_ptr(), ends.data_ptr(), p24.data_ptr() if sites else None,
              site4.data_ptr() if sites else None, gpu._stream())
    t = data[28*m:44*m].reshape(4, m, 4)
    got = host(ends).reshape(3, 2*m, 4)
    order = [(s, b, end) for s in range(n) for b in range(m) for end in (0, 1) if (cpu.i, cpu.j)[end][b] == s]
    assert len(order) == 2*m
    rows = {}
    for k in range(2*m):
        rows.setdefault(tuple(np.abs(got[0, k, :3])), []).append(k)
    a = np.float32(alpha)
    for s, b, end in order:
        sign = np.float32(1 - 2*end)
        want = np.concatenate((sign*t[0, b, :3], t[1 + end, b, :3]))
        near = [k for k in rows[tuple(np.abs(t[0, b, :3]))]
                if np.array_equal(np.concatenate((got[0, k], got[1, k, :2])), want)]
        assert len(near) == 1
        k = near[0]
        assert got[1, k, 3] == a*t[0, b, 3]
        assert np.array_equal(got[2, k, :3], a*np.array([t[1, b, 3], t[2, b, 3], t[3, b, 0]]))
        assert got[2, k, 3].view(np.int32) == (cpu.j, cpu.i)[end][b]
    if sites:
        r, c = np.triu_indices(6)
        assert np.array_equal(host(p24).reshape(n, 24)[:, :21], P[:, r, c])
        fixed = host(gpu.fixed).astype(bool)
        want = np.where(fixed[:, None], [1, 1, 0, 0], np.stack((mass[:, 0], mass[:, 3], np.ones(n), np.zeros(n)), 1))
        assert np.array_equal(host(site4).reshape(n, 4), want.astype(np.float32))
    else:
        assert (host(p24) == -7).all() and (host(site4) == -7).all()


def test_conversions_equal_the_casts():
    """Every class of value: normal, ties, carries into the exponent, both ends of float32's range,
    subnormal, zero, infinite and not a number; the same bits as the casts."""
    import torch
    from dpf_gb300 import _lib
    rng = np.random.default_rng(5)
    bits = rng.integers(0, 2**64, 40000, dtype=np.uint64)
    near = (rng.integers(890, 1155, 40000).astype(np.uint64) << np.uint64(52)) | (bits & np.uint64(0x800fffffffffffff))
    tie = (near & ~np.uint64(0x1fffffff)) | np.uint64(0x10000000)
    edge = np.array([0., -0., np.inf, -np.inf, np.nan, 1., 2.**-126, 2.**-126*(1 - 2.**-25), 2.**-149, 2.**-150, 2.**-1074,
                     3.4028234663852886e38, 3.4028235677973366e38, 1e300, -1e-300, 1 - 2.**-25, 1 + 2.**-24])
    v = np.concatenate((bits.view(np.float64), near.view(np.float64), tie.view(np.float64),
                        (tie + np.uint64(1)).view(np.float64), (tie - np.uint64(1)).view(np.float64), edge))
    stream = torch.cuda.current_stream().cuda_stream
    d = torch.as_tensor(v).cuda()
    out = torch.empty(len(v), dtype=torch.float32, device='cuda')
    _lib.call('dpf_to_float', len(v), d.data_ptr(), out.data_ptr(), stream)
    with np.errstate(over='ignore', invalid='ignore', under='ignore'):
        want = v.astype(np.float32)
    got = host(out)
    number = ~np.isnan(v)
    assert np.array_equal(got[number].view(np.uint32), want[number].view(np.uint32)) and np.isnan(got[~number]).all()

    # s = P r / units with P = 1, one entry a site: (double)(float)r
    n = len(v)
    r = torch.zeros((n, 6), dtype=torch.float64, device='cuda')
    at = torch.arange(n, device='cuda') % 6
    r[torch.arange(n, device='cuda'), at] = d
    eye = torch.eye(6, dtype=torch.float32, device='cuda').repeat(n, 1, 1)
    units, scaled = torch.ones((n, 6), dtype=torch.float32, device='cuda'), torch.empty_like(r)
    _lib.call('dpf_mixed_scale_residual', n, eye.data_ptr(), units.data_ptr(), r.data_ptr(), scaled.data_ptr(), None,
              None, stream)
    got = host(scaled[torch.arange(n, device='cuda'), at])
    assert np.array_equal(got[number], want[number].astype(np.float64)) and np.isnan(got[~number]).all()


@pytest.mark.parametrize('n,m', [(2, 1), (17, 127), (40, 129), (300, 2049)])
@pytest.mark.parametrize('unit', [True, False])
@pytest.mark.parametrize('shift', [0, 1])
def test_float32_jacobian_vector(n, m, unit, shift):
    """J d of the float32 passes against the float64 product, for committed normals that are unit vectors and
    not, and for float32 rows aligned to 8 bytes and not (shift).  A bond's wrench takes some 60 roundings of
    2^-24 to its terms, which a site adds with random signs: 1e-6 of the whole."""
    import torch
    import dpf_gb300
    from dpf_gb300 import _lib
    rng = np.random.default_rng(n)
    side = int(np.ceil(n**(1/3)))
    points = np.stack(np.meshgrid(*[np.arange(side)]*3, indexing='ij'), -1).reshape(-1, 3)[:n] + rng.uniform(-.2, .2, (n, 3))
    i = rng.integers(0, n, m)
    pairs = np.stack((i, (i + rng.integers(1, n, m)) % n), 1)
    given = points[pairs].mean(1) + rng.normal(0, .1, (m, 3))
    s = dpf_gb300.MixedNewtonBonds(points, rng.uniform(.3, .6, n), pairs, rng.uniform(.5, 1., m),
                                   rng.uniform(.5, 2., n), np.arange(n) % 5 == 3, contacts=given)
    for name, shape in (('fn', m), ('mt', m), ('fs', (m, 3)), ('mb', (m, 3))):
        setattr(s, name, s.tensor(rng.normal(size=shape)))
    if not unit:
        s.normal = s.normal*s.tensor(1 + .1*rng.random((m, 1)))
    dt, y, d = 1e-1, s.tensor(rng.normal(0, .02, (n, 6))), s.tensor(rng.normal(size=(n, 6)))
    y[s.fixed] = 0.
    d[s.fixed] = 0.
    external = torch.zeros_like(y)
    s._v = s._vec(s.v).clone()
    s._step_begin(dt, external)
    s._iteration_residual(y, dt, external)
    y32, d32 = (torch.empty(6*n + 1, dtype=torch.float32, device=s.device)[shift:shift + 6*n] for _ in range(2))
    y32.copy_(y.reshape(-1))
    out = torch.empty_like(y)
    _lib.call('dpf_mixed_jacobian_vector', ctypes.byref(s._graph), s._bond_data.data_ptr(), y32.data_ptr(),
              d.data_ptr(), s._mass32.data_ptr(), s.fixed.data_ptr(), dt, None, None, out.data_ptr(), d32.data_ptr(),
              s._wrench32.data_ptr(), None, None, s._stream())
    want = dpf_gb300.NewtonBonds.jacobian_vector(s, y, d, dt, external)
    assert float(torch.linalg.vector_norm(out - want)) <= 1e-6*float(torch.linalg.vector_norm(want))


@pytest.mark.parametrize('m', [2, 5])
@pytest.mark.parametrize('shift', [1, 2, 4])
def test_end_pcg_alignment(m, shift):
    """The PCG's first and last site rows in wide accesses against scalar ones (arrays shifted by floats):
    the same arithmetic, the same bits."""
    import torch
    import dpf_gb300
    from dpf_gb300 import _lib
    foam = dpf_gb300.jittered_lattice_foam(m, seed=m)
    s = dpf_gb300.MixedNewtonBonds(*(foam[k] for k in ('points', 'radii', 'pairs', 'areas', 'masses', 'fixed')),
                                   young=foam['young'], shear=foam['shear'])
    load = s.tensor(dpf_gb300.gravity_load(foam)*4.)
    s.step(2e-3, load, tolerance=1e-6)
    s._pack_ends(2e-3)
    n, rng = s.n_sites, np.random.default_rng(m)
    vector = torch.as_tensor(rng.normal(size=6*n).astype(np.float32)).to(s.device)
    outs = []
    for k in (0, shift):
        place = lambda t: torch.cat((torch.zeros(k, dtype=torch.float32, device=s.device), t.reshape(-1)))[k:]
        block, units, v = place(s._block32), place(s._units32), place(vector)
        out = place(torch.zeros_like(vector))
        s._status.zero_()
        _lib.call('dpf_end_precondition_f32', ctypes.byref(s._graph), s._ends.data_ptr(), s._site4.data_ptr(),
                  s.fixed.data_ptr(), block.data_ptr(), s._p24.data_ptr(), units.data_ptr(), v.data_ptr(), .03, 80,
                  out.data_ptr(), s._inner.data_ptr(), s._tiled_workspace.data_ptr(), s._tiled_partials.data_ptr(),
                  s._barrier.data_ptr(), s._status.data_ptr(), 0, s._stream())
        assert int(s._status[0]) == 0
        outs.append(host(out))
    assert np.array_equal(*outs) and np.abs(outs[0]).max() > 0


@pytest.mark.parametrize('m', [2, 3, 5, 16, 21, 22])
@pytest.mark.parametrize('masked', [False, True])
def test_pcg_of_small_graphs(m, masked):
    """The PCG with a group of lanes a site (the (8, 2) shape up to 9728 sites: 21^3, not 22^3; the (4, 2)
    shape up to 19456: both) against the looping kernel after six iterations: a float32 operator (2e-6) applied six times, 2e-5; with requests
    whose ends are skipped."""
    import torch
    import dpf_gb300
    from dpf_gb300 import _lib
    foam = dpf_gb300.jittered_lattice_foam(m, seed=m)
    s = dpf_gb300.MixedNewtonBonds(*(foam[k] for k in ('points', 'radii', 'pairs', 'areas', 'masses', 'fixed')),
                                   young=foam['young'], shear=foam['shear'])
    load = s.tensor(dpf_gb300.gravity_load(foam)*4.)
    s.step(2e-3, load, tolerance=1e-6)
    s._pack_ends(2e-3)
    n, rng = s.n_sites, np.random.default_rng(m)
    vector = rng.normal(size=(n, 6))
    seg = np.zeros(n, np.int32)
    active = np.ones(2, np.uint8)
    if masked:        # the second half of the sites frozen: zero rows, ends skipped
        seg[n//2:] = 1
        active[1] = 0
        vector[n//2:] = 0.
    vector, seg, active = s.tensor(vector), torch.as_tensor(seg).to(s.device), torch.as_tensor(active).to(s.device)
    outs, counts = [], []
    for variant in (0, 4, 5):
        out, inner = torch.full_like(vector, np.nan), torch.zeros(1, dtype=torch.int32, device=s.device)
        s._status.zero_()
        _lib.call('dpf_end_precondition', ctypes.byref(s._graph), s._ends.data_ptr(), s._site4.data_ptr(),
                  s.fixed.data_ptr(), s._block32.data_ptr(), s._p24.data_ptr(), s._units32.data_ptr(),
                  vector.data_ptr(), 0., 6, out.data_ptr(), inner.data_ptr(), s._tiled_workspace.data_ptr(),
                  s._tiled_partials.data_ptr(), s._barrier.data_ptr(), s._status.data_ptr(),
                  seg.data_ptr() if masked else None, active.data_ptr() if masked else None, variant, s._stream())
        assert int(s._status[0]) == 0
        outs.append(host(out))
        counts.append(int(inner[0]))
    for out, count in zip(outs[1:], counts[1:]):
        assert counts[0] == count
        assert np.linalg.norm(outs[0] - out) <= 2e-5*np.linalg.norm(outs[0])
        assert not masked or not out[n//2:].any()


@pytest.mark.parametrize('n,variant', [(1, 5), (9728, 5), (9729, 4), (19456, 4), (19457, 0), (10**7, 0)])
def test_shape_by_site_count(n, variant):
    from dpf_gb300 import _lib
    assert _lib.load().dpf_end_variant_for(n) == variant
