"""The adjoint's bond passes against torch.autograd of the same trial written in
torch (float64, CPU): input adjoints for given output adjoints, and the local
Jacobians through <lam, J d> = <J^T lam, d>, on graphs whose bond counts
straddle warps and blocks, with classical and given contacts, committed normals
that are unit vectors and not.  The derivatives are sums of a few hundred
products of order one: 1e-10 relative."""
import ctypes

import numpy as np
import pytest

from tests.helpers import host
from tests.test_gpu_float64_passes import DT, _pair

pytestmark = pytest.mark.gpu


def _carry(torch, n0, n1, spin, v):
    cross = lambda a, b: torch.linalg.cross(a, b, dim=1)
    dot = lambda a, b: (a*b).sum(1, keepdim=True)
    k, c = cross(n0, n1), dot(n0, n1).clamp(-1, 1)
    b = n0 + n1
    angle = dot(spin, b/torch.linalg.vector_norm(b, dim=1, keepdim=True).clamp_min(1e-12))
    v = v + cross(k, v) + cross(k, cross(k, v))/(1 + c)
    return torch.cos(angle)*v + torch.sin(angle)*cross(n1, v) + (1 - torch.cos(angle))*dot(n1, v)*n1


def _trial(torch, cpu, y, x, normal, offset, fn, fs, mt, mb, k):
    """Wrenches [F, T_i, T_j] and end history [normal, offset, fn, fs, mt, mb] of every bond."""
    cross = lambda a, b: torch.linalg.cross(a, b, dim=1)
    dot = lambda a, b: (a*b).sum(1, keepdim=True)
    i, j = torch.as_tensor(cpu.i), torch.as_tensor(cpu.j)
    rad = torch.as_tensor(.5*(cpu.radii[cpu.i] - cpu.radii[cpu.j]))[:, None]
    unit = lambda d: d/torch.linalg.vector_norm(d, dim=1, keepdim=True)
    u, w = y[:, :3], y[:, 3:]
    mid, end = x + .5*u, x + u
    n, ne = unit(mid[j] - mid[i]), unit(end[j] - end[i])
    spin = .25*(w[i] + w[j])
    off, fs0, mb0 = (_carry(torch, normal, n, spin, a) for a in (offset, fs, mb))
    contact = .5*(mid[i] + mid[j]) + rad*n + off
    ri, rj = contact - mid[i], contact - mid[j]
    du, dw = u[j] - u[i] + cross(w[j], rj) - cross(w[i], ri), w[j] - w[i]
    dn, tw = dot(du, n), dot(dw, n)
    fn1, mt1 = fn[:, None] + k[:, :1]*dn, mt[:, None] + k[:, 3:]*tw
    fs1, mb1 = fs0 + k[:, 1:2]*(du - dn*n), mb0 + k[:, 2:3]*(dw - tw*n)
    f, c = .5*(fn[:, None] + fn1)*n + .5*(fs0 + fs1), .5*(mt[:, None] + mt1)*n + .5*(mb0 + mb1)
    wrench = torch.cat((f, cross(ri, f) + c, -cross(rj, f) - c), 1)
    return wrench, torch.cat((ne, _carry(torch, n, ne, spin, off), fn1, _carry(torch, n, ne, spin, fs1), mt1,
                              _carry(torch, n, ne, spin, mb1)), 1)


@pytest.mark.parametrize('n,m', [(2, 1), (17, 33), (65, 255)])
@pytest.mark.parametrize('contacts,unit', [(False, True), (True, True), (True, False)])
@pytest.mark.parametrize('end', [False, True])
def test_input_adjoints_and_transposed_product(n, m, contacts, unit, end):
    import torch
    from dpf_gb300 import _lib
    gpu, cpu, rng = _pair(n, m, contacts, unit, seed=n)
    t = lambda a: torch.as_tensor(np.array(a, dtype=np.float64))
    y = rng.normal(0, .02, (n, 6))
    inputs = [t(a).requires_grad_(True) for a in (
        y, cpu.x, cpu.normal, cpu.offset, cpu.fn, cpu.fs, cpu.mt, cpu.mb,
        np.stack((cpu.kn, cpu.ks, cpu.kb, cpu.kt), 1))]
    lam, end_bar, coef = rng.normal(size=(n, 6)), rng.normal(size=(m, 14)), .7
    wrench, history = _trial(torch, cpu, *inputs)
    i, j = cpu.i, cpu.j
    wrench_bar = coef*np.concatenate((lam[i, :3] - lam[j, :3], lam[i, 3:], lam[j, 3:]), 1)
    total = (wrench*t(wrench_bar)).sum() + ((history*t(end_bar)).sum() if end else 0.)
    want = torch.autograd.grad(total, inputs, allow_unused=True)

    lib, g = _lib.load(), gpu.tensor
    hist, stiff, y_bar, x_bar = (torch.zeros(s, dtype=torch.float64, device=gpu.device)
                                 for s in ((m, 14), (m, 4), (n, 6), (n, 3)))
    slots = torch.empty(lib.dpf_adjoint_slot_doubles(m), dtype=torch.float64, device=gpu.device)
    y_d, lam_d, end_d = g(y), g(lam), g(end_bar)
    args = (ctypes.byref(gpu._graph), ctypes.byref(gpu._stiffness_struct()), ctypes.byref(gpu._history_struct()))
    _lib.call('dpf_adjoint_bond_vjp', *args, y_d.data_ptr(), lam_d.data_ptr(), coef,
              end_d.data_ptr() if end else None, 1, hist.data_ptr(), stiff.data_ptr(), y_bar.data_ptr(),
              x_bar.data_ptr(), slots.data_ptr(), gpu._stream())
    got = [y_bar, x_bar, hist[:, 0:3], hist[:, 3:6], hist[:, 6], hist[:, 7:10], hist[:, 10], hist[:, 11:14], stiff]
    for name, a, b in zip(('y', 'x', 'normal', 'offset', 'fn', 'fs', 'mt', 'mb', 'k'), got, want):
        assert np.linalg.norm(host(a) - b.numpy()) <= 1e-10*max(1., float(b.norm())), name

    jac = torch.empty(lib.dpf_adjoint_jacobian_doubles(m), dtype=torch.float64, device=gpu.device)
    _lib.call('dpf_adjoint_local_jacobian', *args, y_d.data_ptr(), jac.data_ptr(), gpu._stream())
    lam[cpu.fixed] = 0.
    lam_d, out = g(lam), torch.empty((n, 6), dtype=torch.float64, device=gpu.device)
    _lib.call('dpf_adjoint_apply_jt', ctypes.byref(gpu._graph), jac.data_ptr(), gpu.mass.data_ptr(),
              gpu.fixed.data_ptr(), DT, lam_d.data_ptr(), out.data_ptr(), slots.data_ptr(), gpu._stream())
    d = rng.normal(size=(n, 6))
    d[cpu.fixed] = 0.
    left, right = (lam*cpu.jacobian_vector(y, d, DT, None)).sum(), (host(out)*d).sum()
    scale = np.linalg.norm(lam)*np.linalg.norm(cpu.jacobian_vector(y, d, DT, None))
    assert abs(left - right) <= 1e-10*scale


@pytest.mark.parametrize('n,m', [(2, 1), (15, 31), (17, 33), (65, 255), (700, 2049)])
def test_scaled_adjoint_system(n, m):
    """The fused operator, multiplier and preconditioner against their definitions (sums of 6: 1e-12; the
    PCG run to 1e-13 on systems of condition below 1e3: 1e-9)."""
    import torch
    from dpf_gb300 import _lib
    gpu, cpu, rng = _pair(n, m, seed=n)
    lib, empty = _lib.load(), lambda *s: torch.empty(s, dtype=torch.float64, device=gpu.device)
    y = gpu.tensor(rng.normal(0, .02, (n, 6)))
    gpu.prepare_scaling(gpu.trial(y), DT)
    units, P, block = gpu.units, gpu.preconditioner, gpu.block
    mu = rng.normal(size=(n, 6))
    mu[cpu.fixed] = 0.
    mu = gpu.tensor(mu)
    jac, slots = empty(max(1, lib.dpf_adjoint_jacobian_doubles(m))), empty(max(1, lib.dpf_adjoint_slot_doubles(m)))
    graph, stream = ctypes.byref(gpu._graph), gpu._stream()
    _lib.call('dpf_adjoint_local_jacobian', graph, ctypes.byref(gpu._stiffness_struct()),
              ctypes.byref(gpu._history_struct()), y.data_ptr(), jac.data_ptr(), stream)
    lam, out, plain = empty(n, 6), empty(n, 6), empty(n, 6)
    _lib.call('dpf_adjoint_operator', graph, jac.data_ptr(), gpu.mass.data_ptr(), gpu.fixed.data_ptr(), P.data_ptr(),
              units.data_ptr(), DT, mu.data_ptr(), out.data_ptr(), lam.data_ptr(), slots.data_ptr(), stream)
    want = (P@(mu/units)[:, :, None])[:, :, 0].contiguous()
    rel = lambda a, b: float(torch.linalg.vector_norm(a - b)/torch.linalg.vector_norm(b).clamp_min(1e-300))
    assert rel(lam, want) <= 1e-12
    _lib.call('dpf_adjoint_multiplier', n, P.data_ptr(), units.data_ptr(), mu.data_ptr(), plain.data_ptr(), stream)
    assert torch.equal(plain, lam)
    _lib.call('dpf_adjoint_apply_jt', graph, jac.data_ptr(), gpu.mass.data_ptr(), gpu.fixed.data_ptr(), DT,
              lam.data_ptr(), plain.data_ptr(), slots.data_ptr(), stream)
    assert rel(out, units*plain) <= 1e-12

    work = empty(lib.dpf_elastic_workspace_doubles(n))
    def pcg(name, block, units, vector, out):
        _lib.call(name, graph, ctypes.byref(gpu._stiffness_struct()), ctypes.byref(gpu._tangent_struct()),
                  gpu.mass.data_ptr(), gpu.fixed.data_ptr(), block.data_ptr(), P.data_ptr(), units.data_ptr(),
                  vector.data_ptr(), DT, 1e-13, 400, out.data_ptr(), gpu._inner.data_ptr(), gpu._wrench.data_ptr(),
                  work.data_ptr(), gpu._barrier.data_ptr(), gpu._status.data_ptr(), stream)
    gpu._status.zero_()
    pcg('dpf_adjoint_precondition', block, units, mu, out)
    identity, ones = torch.eye(6, dtype=block.dtype, device=gpu.device).repeat(n, 1, 1), torch.ones_like(units)
    pcg('dpf_elastic_precondition', identity, ones, mu/units, plain)
    assert int(gpu._status[0]) == 0
    assert rel(out, units*(block@plain[:, :, None])[:, :, 0]) <= 1e-9


@pytest.mark.parametrize('length,j', [(2, 0), (6, 4), (257, 8), (257, 62), (70001, 31)])
def test_fused_arnoldi_step(length, j):
    """One cooperative launch against the four-pass step: the same column and next row (dot products of
    unit rows, 1e-12 of |w|; the next row is divided by a remainder of the order of |w|)."""
    import torch
    from dpf_gb300 import _lib
    lib, dev = _lib.load(), torch.device('cuda')
    rng = np.random.default_rng(length + j)
    rows = np.linalg.qr(rng.normal(size=(length, j + 1)))[0].T
    got = []
    for name in ('dpf_arnoldi_cgs2', 'dpf_arnoldi_cgs2_fused'):
        basis = torch.zeros((j + 2, length), dtype=torch.float64, device=dev)
        basis[:j + 1] = torch.as_tensor(rows)
        w = torch.as_tensor(np.random.default_rng(j).normal(size=length)).to(dev)
        h = torch.zeros(72, dtype=torch.float64, device=dev)
        partials = torch.zeros(max(lib.dpf_partials_doubles(), lib.dpf_newton64_partials_doubles()),
                               dtype=torch.float64, device=dev)
        barrier = torch.ones(4, dtype=torch.int32, device=dev)
        barrier[2:] = 0
        extra = () if name == 'dpf_arnoldi_cgs2' else (barrier.data_ptr(), barrier[2:].data_ptr())
        _lib.call(name, length, basis.data_ptr(), length, j, w.data_ptr(), h.data_ptr(), partials.data_ptr(), *extra,
                  torch.cuda.current_stream(dev).cuda_stream)
        assert int(barrier[2]) == 0
        got.append((host(h), host(basis), host(w)))
    size = np.sqrt(length)
    (h0, b0, w0), (h1, b1, w1) = got
    assert np.abs(h0 - h1).max() <= 1e-12*size and np.abs(w0 - w1).max() <= 1e-12*size
    assert h0[j + 1] > 1e-3*size
    assert np.abs(b0 - b1).max() <= 1e-12*size/h0[j + 1]*10


@pytest.mark.parametrize('n', [1, 16, 17, 700])
def test_adjoint_site_passes(n):
    """The joined site passes against the same sums in torch (one or two roundings of each: 1e-15)."""
    import torch
    from dpf_gb300 import _lib
    dev, dt = torch.device('cuda'), 3e-3
    rng = np.random.default_rng(n)
    t = lambda *s: torch.as_tensor(rng.normal(size=s)).to(dev)
    x_bar, v_bar, g, units, mass, lam, v = t(n, 3), t(n, 6), t(n, 3), t(n, 6), t(n, 6), t(n, 6), t(n, 6)
    fixed = torch.as_tensor(np.arange(n) % 3 == 1).to(dev)
    y_bar, x_next, v_next, rhs, load = (torch.full(s, np.nan, dtype=torch.float64, device=dev)
                                        for s in ((n, 6), (n, 3), (n, 6), (n, 6), (n, 6)))
    p, stream = (lambda a: a.data_ptr()), torch.cuda.current_stream(dev).cuda_stream
    _lib.call('dpf_adjoint_commit_map', n, dt, p(x_bar), p(v_bar), p(g), p(y_bar), p(x_next), p(v_next), stream)
    want = (2/dt)*v_bar
    want[:, :3] += x_bar
    close = lambda a, b: bool((a - b).abs().max() <= 1e-15*b.abs().max())
    assert close(y_bar, want) and torch.equal(x_next, x_bar + g) and torch.equal(v_next, -v_bar)
    _lib.call('dpf_adjoint_rhs', n, p(y_bar), p(units), p(fixed), p(rhs), stream)
    assert torch.equal(rhs, torch.where(fixed[:, None], torch.zeros_like(rhs), units*y_bar))
    v0 = v.clone()
    _lib.call('dpf_adjoint_loads', n, dt, p(mass), p(lam), p(load), p(v), stream)
    assert close(load, .5*dt*dt*lam) and close(v, v0 + dt*mass*lam)
