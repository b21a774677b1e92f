"""Performance cases: the work that users of this package have it do.

Every case is one call (or one step) of a public entry point on a synthetic
jittered-lattice power foam of the kind the tests and the benchmark use: sites
in Morton order, about 7.4 bonds per site, one bond list sorted by endpoints.
The bond graph is drawn on the device (lattice neighbours, one diagonal per
lattice face and one or two per lattice cube) instead of triangulated on the
host, so that a 1.4M-site foam is ready in well under a second.

The float64 forms return the state they compute as it is.  The mixed and the
served form compute their velocities with float32 bond sweeps to a stated
relative accuracy of 1e-6; their programs read positions and rotations in
float64 and velocities in float32, and so do these cases.
"""
import ctypes
import math

import numpy as np
import torch

import dpf_gb300
from dpf_gb300 import _lib, serving

F64 = torch.float64
DEVICE = 'cuda'

FORMS = ('newton', 'mixed', 'jacobian', 'hvp', 'linear', 'energy', 'adjoint', 'served')


def _case(name, form, nx, ny, nz, **options):
    """contacts: bonds with given contact points (nonzero offsets) instead of the
    classical ones; preconditioning: of the Newton system; steps: of a
    differentiated rollout; requests: in a served batch."""
    case = dict(name=name, form=form, nx=nx, ny=ny, nz=nz, young=4e5, dt=1e-3, contacts=False,
                preconditioning='elastic', steps=1, requests=1)
    case.update(options)
    return case


def listed():
    return [
        # The drop-in float64 solver: one implicit step of a trajectory.  A specimen of
        # a few hundred cells (the checks' and demos' size), where launches and host
        # reads count, ...
        _case('newton_512', 'newton', 8, 8, 8),
        # ... a ragged body of tens of thousands of cells with given contact points,
        _case('newton_37k', 'newton', 41, 33, 27, contacts=True),
        # ... and the benchmark's 64^3 foam in the plain form.
        _case('newton_262k', 'newton', 64, 64, 64),
        # The mixed-precision form, same step: interactive size, the benchmark's
        # headline foam, and a large one.
        _case('mixed_4k', 'mixed', 16, 16, 16),
        _case('mixed_262k', 'mixed', 64, 64, 64),
        _case('mixed_1400k', 'mixed', 112, 112, 112),
        # One float64 Jacobian product at a prestressed state, as a caller with its own
        # Krylov solver uses it (odd sizes).
        _case('jacobian_101k', 'jacobian', 47, 45, 48, contacts=True),
        # One float32 Hessian-vector product of the elastic operator, the benchmark's
        # HVP workload.
        _case('hvp_262k', 'hvp', 64, 64, 64),
        # The stress-free linear model: one implicit-midpoint step.
        _case('linear_30k', 'linear', 31, 31, 31),
        # The energy law: forces and torques of a deformed foam, as an explicit
        # integrator calls them every substep.
        _case('energy_125k', 'energy', 50, 50, 50),
        # Inverse material fit: forward rollout and the adjoint's gradients.
        _case('adjoint_8k', 'adjoint', 20, 20, 20, steps=3, dt=2e-3, young=1e5),
        # A served batch of requests of uneven size.
        _case('served_16', 'served', 10, 10, 32, requests=16),
    ]


def draw(rng):
    """A case of the same ranges, never larger than the listed ones of its form."""
    form = rng.choice(FORMS)
    low, high = dict(newton=(300, 200000), mixed=(300, 900000), jacobian=(300, 240000), hvp=(2000, 900000),
                     linear=(300, 100000), energy=(300, 240000), adjoint=(300, 8000), served=(300, 3200))[form]
    sites = math.exp(rng.uniform(math.log(low), math.log(high)))
    side = sites**(1/3)
    nx, ny = (max(4, round(side*math.exp(rng.uniform(-.3, .3)))) for _ in range(2))
    nz = max(4, round(sites/(nx*ny)))
    return {k: v for k, v in _case(
        '', form, nx, ny, nz, young=math.exp(rng.uniform(math.log(1e5), math.log(1e6))),
        dt=rng.choice((5e-4, 1e-3)), contacts=form not in ('served', 'adjoint') and rng.random() < .4,
        preconditioning='block' if form == 'newton' and sites < 20000 and rng.random() < .25 else 'elastic',
        steps=rng.choice((2, 3)) if form == 'adjoint' else 1,
        requests=rng.choice((3, 7, 16)) if form == 'served' else 1).items() if k != 'name'}


# ---- inputs ---------------------------------------------------------------------

def _foam(nx, ny, nz, seed, young, contacts):
    """Constructor arguments (host arrays) of a jittered nx x ny x nz foam."""
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
    rand = lambda *shape: torch.rand(shape, generator=gen, device=DEVICE, dtype=F64)
    dims = (nx, ny, nz)
    h = 1./max(dims)
    cell = torch.stack(torch.meshgrid(*(torch.arange(d, device=DEVICE) for d in dims), indexing='ij'), -1).reshape(-1, 3)
    code = torch.zeros(len(cell), dtype=torch.int64, device=DEVICE)
    for bit in range(max(dims).bit_length()):
        for axis in range(3):
            code |= ((cell[:, axis] >> bit) & 1) << (3*bit + axis)
    order = torch.argsort(code)
    n = len(cell)
    rank = torch.empty(n, dtype=torch.int64, device=DEVICE)
    rank[order] = torch.arange(n, device=DEVICE)
    rank = rank.view(nx, ny, nz)

    pairs = []

    def corners(axes):
        """Minimum corners of every lattice edge / face / cube spanned by ``axes``."""
        return cell[torch.stack([cell[:, a] < dims[a] - 1 for a in axes]).all(0)]

    def connect(a, b):
        pairs.append(torch.stack((rank[tuple(a.T)], rank[tuple(b.T)]), 1))
    unit = torch.eye(3, dtype=torch.int64, device=DEVICE)
    for a in range(3):
        c = corners((a,))
        connect(c, c + unit[a])
    for a, b in ((0, 1), (0, 2), (1, 2)):            # one of the two diagonals of each face
        c = corners((a, b))
        flip = (rand(len(c)) < .5)[:, None]
        connect(torch.where(flip, c + unit[a], c), torch.where(flip, c + unit[b], c + unit[a] + unit[b]))
    c = corners((0, 1, 2))                           # one or two of the four diagonals of each cube
    first = (rand(len(c))*4).long()
    second = (first + 1 + (rand(len(c))*3).long()) % 4
    both = torch.argsort(rand(len(c)))[:round(.46*len(c))]      # as many for every seed
    for which, where in ((first, slice(None)), (second, both)):
        start, stop = c.clone(), c + 1
        for a in range(3):                           # diagonal k starts at the corner raised along axis k - 1
            up = which == a + 1
            start[up, a] += 1
            stop[up, a] -= 1
        connect(start[where], stop[where])
    pairs = torch.cat(pairs).sort(1).values
    pairs = pairs[torch.argsort(pairs[:, 0]*n + pairs[:, 1])]

    points = (cell[order] + .5 + .4*(rand(n, 3) - .5))*h
    areas = (.5 + .5*rand(len(pairs)))*h*h
    radii = torch.full((n,), .5*h, dtype=F64, device=DEVICE)
    given = None
    if contacts:                                     # uneven cells: contact points off the classical ones
        radii = h*(.4 + .2*rand(n))
        i, j = pairs.T
        d = points[j] - points[i]
        normal = d/torch.linalg.vector_norm(d, dim=1, keepdim=True)
        given = .5*(points[i] + points[j]) + .5*(radii[i] - radii[j])[:, None]*normal + .1*h*(rand(len(pairs), 3) - .5)
    host = lambda t: None if t is None else t.cpu().numpy()
    fixed = cell[order][:, 2] < max(1, round(.05*nz))
    return dict(points=host(points), radii=host(radii), pairs=host(pairs), areas=host(areas),
                masses=np.full(n, 1000.*h**3), fixed=host(fixed), contacts=host(given), young=float(young),
                shear=float(young)/2.6)


def _weight(foam):
    load = np.zeros((len(foam['points']), 6))
    load[:, 2] = -9.81*foam['masses']
    load[foam['fixed']] = 0.
    return load


def _velocity(foam, seed):
    """A smooth velocity field of about 0.02 m/s with slow spins, zero on fixed sites."""
    rng = np.random.default_rng(int(seed))
    x = torch.as_tensor(foam['points'], device=DEVICE)
    k = torch.as_tensor(rng.uniform(1., 4., (6, 3)), device=DEVICE)
    v = torch.sin(x@k.T*2 + torch.as_tensor(rng.uniform(0., 6.28, 6), device=DEVICE))
    v = v*torch.tensor([.02, .02, .02, .1, .1, .1], dtype=F64, device=DEVICE)
    v[torch.as_tensor(foam['fixed'], device=DEVICE)] = 0.
    return v


def _prestress(s, seed):
    """A committed history with forces of about 1% strain."""
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed) + 1)
    noise = lambda like: torch.randn(like.shape, generator=gen, device=DEVICE, dtype=F64)
    h = s.radii.max()
    s.fn = s.kn*h*.02*noise(s.kn)
    s.mt = s.kt*.01*noise(s.kt)
    across = lambda t: t - (t*s.normal).sum(1, keepdim=True)*s.normal
    s.fs = (s.ks*h*.01)[:, None]*across(noise(s.normal))
    s.mb = (s.kb*.01)[:, None]*across(noise(s.normal))


def _solver(cls, foam):
    return cls(foam['points'], foam['radii'], foam['pairs'], foam['areas'], foam['masses'], foam['fixed'],
               contacts=foam['contacts'], young=foam['young'], shear=foam['shear'], device=DEVICE)


def _displacement(foam, seed, size):
    """A smooth increment of ``size`` spacings and radians, zero on fixed sites."""
    h = 2*float(np.max(foam['radii']))
    scale = torch.tensor([h, h, h, 1., 1., 1.], dtype=F64, device=DEVICE)*size
    return _velocity(foam, seed + 2)*scale/torch.tensor([.02]*3 + [.1]*3, dtype=F64, device=DEVICE)


def _direction(foam, seed):
    """A rough vector as a Krylov method meets it (lengths in spacings), zero on fixed sites."""
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed) + 3)
    d = torch.randn((len(foam['points']), 6), generator=gen, device=DEVICE, dtype=F64)
    d[:, :3] *= 2*float(np.max(foam['radii']))
    d[torch.as_tensor(foam['fixed'], device=DEVICE)] = 0.
    return d


def _request_foams(case, seed):
    """Foams of nx x ny x k lattices, k spread over the logarithm up to nz, and their loads."""
    rng = np.random.default_rng(int(seed))
    out = []
    for index in range(case['requests']):
        k = round(4*(max(5, case['nz'])/4)**((index + .5)/case['requests']))
        foam = _foam(case['nx'], case['ny'], k, int(rng.integers(1 << 31)),
                     case['young']*math.exp(rng.uniform(-1., 1.)), False)
        load = _weight(foam)
        top = foam['points'][:, 2] > foam['points'][:, 2].max() - .6*2*foam['radii'][0]
        load[top & ~foam['fixed'], 2] -= foam['young']*.02*(2*foam['radii'][0])**2
        out.append((foam, load))
    return out


def prepare(case, seed):
    form, dt = case['form'], case['dt']
    state = dict(case, foam=None)
    if form == 'served':
        state['requests'] = _request_foams(case, seed)
        state['service'] = serving.Service(device=DEVICE, hbm_budget=6e9, max_batch_sites=100_000, tolerance=1e-6)
        return state
    foam = state['foam'] = _foam(case['nx'], case['ny'], case['nz'], seed, case['young'], case['contacts'])
    load = torch.as_tensor(_weight(foam), device=DEVICE)
    state['load'] = load
    if form in ('newton', 'mixed', 'jacobian', 'hvp'):
        s = state['solver'] = _solver(dpf_gb300.NewtonBonds if form in ('newton', 'jacobian') else
                                      dpf_gb300.MixedNewtonBonds, foam)
        s.v = _velocity(foam, seed)
    if form == 'jacobian':
        _prestress(s, seed)
        state['y'] = _displacement(foam, seed, 5e-3)
        state['direction'] = _direction(foam, seed)
    elif form == 'hvp':
        s.step(dt, load, tolerance=1e-6)
        s._pack_ends(dt)
        state['q'] = _direction(foam, seed).float()
        state['out'] = torch.empty_like(state['q'])
    elif form == 'linear':
        contacts = foam['contacts']
        if contacts is None:
            i, j = foam['pairs'].T
            contacts = .5*(foam['points'][i] + foam['points'][j])
        s = state['solver'] = dpf_gb300.LinearBonds(
            foam['points'], foam['radii'], foam['pairs'], foam['areas'], contacts, foam['masses'], foam['fixed'],
            young=foam['young'], shear=foam['shear'], device=DEVICE)
        s.v = _velocity(foam, seed)
    elif form == 'energy':
        i, j = foam['pairs'].T
        contacts = foam['contacts'] if foam['contacts'] is not None else .5*(foam['points'][i] + foam['points'][j])
        state['law'] = dpf_gb300.EnergyFoam(dict(foam, contacts=contacts), volume=False, young=foam['young'],
                                            shear=foam['shear'], device=DEVICE)
        turn = _displacement(foam, seed, .05)
        state['theta'] = .1*_velocity(foam, seed + 5)[:, :4]/.02
        state['x'] = torch.as_tensor(foam['points'], device=DEVICE) + turn[:, :3]
        half = .5*torch.linalg.vector_norm(turn[:, 3:], dim=1, keepdim=True)
        state['q'] = torch.cat((torch.cos(half), .5*turn[:, 3:]*torch.sinc(half/math.pi)), 1)
    elif form == 'adjoint':
        m = state['model'] = dpf_gb300.DifferentiableBonds(
            points=foam['points'], radii=foam['radii'], pairs=foam['pairs'], areas=foam['areas'],
            masses=foam['masses'], fixed=foam['fixed'], young=foam['young'], shear=foam['shear'], device=DEVICE,
            checkpoint_every=2)
        gen = torch.Generator(device=DEVICE).manual_seed(int(seed) + 3)
        factor = torch.exp(.3*torch.randn(len(foam['pairs']), generator=gen, device=DEVICE, dtype=F64))
        state['stiffness'] = (m.base_stiffness*factor[:, None]).requires_grad_(True)
        state['loads'] = load[None].repeat(case['steps'], 1, 1).requires_grad_(True)
        initial = list(m.initial_state())
        initial[1] = _velocity(foam, seed)
        initial[0].requires_grad_(True)
        initial[1].requires_grad_(True)
        state['initial'] = tuple(initial)
        ramp = torch.arange(case['steps'] + 1, device=DEVICE, dtype=F64)[:, None, None]/case['steps']
        state['target'] = initial[0].detach() + ramp*_displacement(foam, seed + 4, 1e-2)[:, :3]
    return state


# ---- one pass -------------------------------------------------------------------

def run(state):
    form = state['form']
    if form == 'newton':
        s = state['solver']
        work, _ = s.step(state['dt'], state['load'], preconditioning=state['preconditioning'])
        return dict(x=s.x, v=s.v, rotation=s.rotation, normal=s.normal, fn=s.fn, fs=s.fs, mt=s.mt, mb=s.mb, work=work)
    if form == 'mixed':
        s = state['solver']
        s.step(state['dt'], state['load'], tolerance=1e-6)
        return dict(x=s.x, v=s.v.float(), rotation=s.rotation)
    if form == 'jacobian':
        return state['solver'].jacobian_vector(state['y'], state['direction'], state['dt'], state['load'])
    if form == 'hvp':
        s = state['solver']
        _lib.call('dpf_end_hvp', ctypes.byref(s._graph), s._ends.data_ptr(), s._site4.data_ptr(),
                  state['q'].data_ptr(), state['out'].data_ptr(), 0, torch.cuda.current_stream().cuda_stream)
        return state['out']
    if form == 'linear':
        s = state['solver']
        work, _ = s.step(state['dt'], state['load'])
        return dict(q=s.q, v=s.v, kq=s.kq, work=work)
    if form == 'energy':
        return state['law'].forces(state['theta'], state['x'], state['q'])
    if form == 'adjoint':
        positions, *_ = state['model'].rollout_bonds(state['stiffness'], state['loads'], state['initial'], state['dt'])
        wanted = (state['stiffness'], state['loads'], state['initial'][0], state['initial'][1])
        grads = torch.autograd.grad(((positions - state['target'])**2).sum(), wanted)
        return dict(positions=positions.detach(), stiffness=grads[0], loads=grads[1], x=grads[2], v=grads[3])
    requests = [serving.Request(arrival=0., rid=k, foam=foam, load=load, dt=state['dt'])
                for k, (foam, load) in enumerate(state['requests'])]
    finished = sorted(state['service'].run(requests), key=lambda r: r.rid)
    return dict(x=torch.cat([r.state['x'] for r in finished]), v=torch.cat([r.state['v'] for r in finished]).float(),
                rotation=torch.cat([r.state['rotation'] for r in finished]))


# ---- what a pass cannot do without ----------------------------------------------

def _size(nx, ny, nz):
    edges = (nx - 1)*ny*nz + nx*(ny - 1)*nz + nx*ny*(nz - 1)
    faces = (nx - 1)*(ny - 1)*nz + (nx - 1)*ny*(nz - 1) + nx*(ny - 1)*(nz - 1)
    return nx*ny*nz, edges + faces + 1.46*(nx - 1)*(ny - 1)*(nz - 1)


def work(case):
    """Each input read once and each output written once; operations of the law
    as it is written down: about 300 per bond and evaluation, 400 per Jacobian
    product, 120 per stiffness product, 500 per site for its 6x6 block.  A step
    is counted with one Newton iteration, two Krylov vectors and twelve CG
    iterations."""
    n, m = _size(case['nx'], case['ny'], case['nz'])
    form = case['form']
    history = 14*8                                # normal, offset, fn, fs, mt, mb
    if form in ('newton', 'mixed', 'served'):
        if form == 'served':                      # k averages about nz/2.6 over its range
            n, m = n*case['requests']/2.6, m*case['requests']/2.6
        sites = (3 + 6 + 9)*16 + 6*8 + 6*8 + 8
        bonds = 16 + 4*8 + 2*history
        return dict(bytes=bonds*m + sites*n, flops=(2*300 + 2*400 + 12*120)*m + (500 + 12*150)*n)
    if form == 'jacobian':
        return dict(bytes=(16 + 4*8 + history)*m + (3 + 1 + 6 + 6 + 6 + 6)*8*n, flops=400*m + 20*n)
    if form == 'hvp':
        return dict(bytes=60*m + 56*n, flops=120*m + 12*n)
    if form == 'linear':
        return dict(bytes=(16 + 13*8)*m + (6*8 + 36 + 6*6)*8*n/2, flops=30*120*m + 30*150*n)
    if form == 'energy':
        return dict(bytes=(16 + 13*8)*m + (4 + 3 + 4 + 6)*8*n, flops=300*m)
    steps = case['steps']
    return dict(bytes=steps*(2*(16 + 4*8 + 2*history)*m + 3*(3 + 6 + 9)*8*n),
                flops=steps*((6*300 + 10*400 + 60*120)*m + (1500 + 60*150)*n))


# ---- the same in 64 bits, in plain torch ----------------------------------------

def _cross(a, b):
    return torch.linalg.cross(a, b, dim=1)


def _dot(a, b):
    return (a*b).sum(1, keepdim=True)


def _carry(n0, n1, spin, vectors):
    """Shortest-arc rotation from n0 to n1, then a spin about n1."""
    axis, cosine = _cross(n0, n1), _dot(n0, n1)
    middle = n0 + n1
    angle = _dot(spin, middle/torch.linalg.vector_norm(middle, dim=1, keepdim=True))
    s, c = torch.sin(angle), torch.cos(angle)
    out = []
    for v in vectors:
        once = _cross(axis, v)
        v = v + once + _cross(axis, once)/(1 + cosine)
        out.append(c*v + s*_cross(n1, v) + (1 - c)*_dot(n1, v)*n1)
    return out


class _Law:
    """The rate law in torch: forces and end history of an increment, the frozen
    tangent's product, and iterations that solve with it to rounding."""

    def __init__(self, foam):
        t = lambda a: torch.as_tensor(a, dtype=F64, device=DEVICE)
        self.points, self.radii, self.fixed = t(foam['points']), t(foam['radii']), torch.as_tensor(foam['fixed'], device=DEVICE)
        self.i, self.j = torch.as_tensor(foam['pairs'], device=DEVICE).T
        m = t(foam['masses'])[:, None]
        self.mass = torch.cat((m.expand(-1, 3), (.4*m*self.radii[:, None]**2).expand(-1, 3)), 1)
        d = self.points[self.j] - self.points[self.i]
        length = torch.linalg.vector_norm(d, dim=1)
        area = t(foam['areas'])
        second = area**2/(4*math.pi)
        E, G = foam['young'], foam['shear']
        self.k = torch.stack((E*area, G*area, E*second, G*2*second), 1)/length[:, None]
        normal, classical = self.geometry(self.points)
        contact = classical if foam['contacts'] is None else t(foam['contacts'])
        self.contact = contact
        zero, none = torch.zeros_like(normal), torch.zeros_like(length)[:, None]
        self.history = (normal, contact - classical, none, zero, none, zero)

    def geometry(self, x):
        xi, xj = x[self.i], x[self.j]
        n = (xj - xi)/torch.linalg.vector_norm(xj - xi, dim=1, keepdim=True)
        return n, .5*(xi + xj) + .5*(self.radii[self.i] - self.radii[self.j])[:, None]*n

    def gather(self, f, ti, tj):
        out = torch.zeros_like(self.mass)
        return out.index_add(0, self.i, torch.cat((f, ti), 1)).index_add(0, self.j, torch.cat((-f, tj), 1))

    def trial(self, x, history, k, y, end=False):
        normal, offset, fn, fs, mt, mb = history
        kn, ks, kb, kt = (k[:, c:c + 1] for c in range(4))
        i, j = self.i, self.j
        u, w = y[:, :3], y[:, 3:]
        n, contact = self.geometry(x + .5*u)
        spin = .25*(w[i] + w[j])
        offset, fs, mb = _carry(normal, n, spin, (offset, fs, mb))
        contact = contact + offset
        ri, rj = contact - (x + .5*u)[i], contact - (x + .5*u)[j]
        du = u[j] - u[i] + _cross(w[j], rj) - _cross(w[i], ri)
        dw = w[j] - w[i]
        stretch, twist = _dot(du, n), _dot(dw, n)
        fn1, mt1 = fn + kn*stretch, mt + kt*twist
        fs1, mb1 = fs + ks*(du - stretch*n), mb + kb*(dw - twist*n)
        f, couple = .5*(fn + fn1)*n + .5*(fs + fs1), .5*(mt + mt1)*n + .5*(mb + mb1)
        force = self.gather(f, _cross(ri, f) + couple, -_cross(rj, f) - couple)
        if not end:
            return force, (n, ri, rj)
        n_end, _ = self.geometry(x + u)
        offset, fs1, mb1 = _carry(n, n_end, spin, (offset, fs1, mb1))
        return (n_end, offset, fn1, fs1, mt1, mb1)

    def residual(self, x, v, history, k, load, dt, y):
        r = self.mass*(y - dt*v) - .5*dt*dt*(self.trial(x, history, k, y)[0] + load)
        return torch.where(self.fixed[:, None], y, r)

    def stiffness(self, q, tangent, k):
        n, ri, rj = tangent
        kn, ks, kb, kt = (k[:, c:c + 1] for c in range(4))
        i, j = self.i, self.j
        du = q[j, :3] - q[i, :3] + _cross(q[j, 3:], rj) - _cross(q[i, 3:], ri)
        dw = q[j, 3:] - q[i, 3:]
        f = ks*du + (kn - ks)*_dot(du, n)*n
        c = kb*dw + (kt - kb)*_dot(dw, n)*n
        return self.gather(-f, -_cross(ri, f) - c, _cross(rj, f) + c)

    def solver(self, tangent, k, dt, tolerance=1e-13):
        """b -> (diag M + dt^2/4 K)^-1 b by CG, identity rows on fixed sites."""
        n, ri, rj = tangent
        kn, ks, kb, kt = (k[:, c:c + 1] for c in range(4))
        a = .25*dt*dt
        diagonal = self.mass.clone()
        for site, r in ((self.i, ri), (self.j, rj)):
            lever = torch.stack([_dot(n, torch.linalg.cross(e.expand_as(r), r, dim=1))[:, 0]
                                 for e in torch.eye(3, dtype=F64, device=DEVICE)], 1)
            turn = ks*(_dot(r, r) - r*r) + (kn - ks)*lever**2 + kb + (kt - kb)*n*n
            diagonal = diagonal.index_add(0, site, a*torch.cat((ks + (kn - ks)*n*n, turn), 1))
        free = (~self.fixed)[:, None].to(F64)

        def solve(b):
            fixed_part = b*(1 - free)
            b = b*free
            x, r = torch.zeros_like(b), b
            z = r/diagonal
            p, rz = z, (r*z).sum()
            limit = tolerance**2*rz
            for k_ in range(600):
                ap = (self.mass*p + a*self.stiffness(p, tangent, k))*free
                step = rz/(p*ap).sum()
                x, r = x + step*p, r - step*ap
                z = r/diagonal
                rz, before = (r*z).sum(), rz
                if k_ % 10 == 9 and not bool(rz > limit):
                    break
                p = z + (rz/before)*p
            return torch.where(torch.isfinite(x), x, torch.zeros_like(x)) + fixed_part
        return solve

    def increment(self, x, v, history, k, load, dt):
        """The y of one implicit-midpoint step, to rounding."""
        y = torch.where(self.fixed[:, None], torch.zeros_like(v), dt*v)
        for _ in range(30):
            solve = self.solver(self.trial(x, history, k, y)[1], k, dt, 1e-8)
            change = solve(self.residual(x, v, history, k, load, dt, y))
            y = y - change
            if bool((change*change).sum() <= 1e-30*(y*y).sum()):
                break
        return y


def _turn(w):
    """exp([w]x) for (N, 3) rotation vectors."""
    a = torch.linalg.vector_norm(w, dim=1)
    s = torch.zeros((len(w), 3, 3), dtype=F64, device=w.device)
    s[:, 0, 1], s[:, 0, 2], s[:, 1, 2] = -w[:, 2], w[:, 1], -w[:, 0]
    s = s - s.transpose(1, 2)
    return (torch.eye(3, dtype=F64, device=w.device) + torch.sinc(a/math.pi)[:, None, None]*s +
            (.5*torch.sinc(a/(2*math.pi))**2)[:, None, None]*(s@s))


class _Implicit(torch.autograd.Function):
    """Zero in value; its gradient carries that of the solution of r(y) = 0."""

    @staticmethod
    def forward(ctx, r, transposed):
        ctx.transposed = transposed
        return torch.zeros_like(r)

    @staticmethod
    def backward(ctx, g):
        return -ctx.transposed(g), None


def _exact_step(foam, load, v, dt):
    law = _Law(foam)
    load = torch.as_tensor(load, device=DEVICE)
    y = law.increment(law.points, v, law.history, law.k, load, dt)
    return law, y, load


def exact(case, seed):
    form, dt = case['form'], case['dt']
    if form == 'served':
        x, v, turn = [], [], []
        for foam, load in _request_foams(case, seed):
            start = torch.zeros((len(load), 6), dtype=F64, device=DEVICE)
            law, y, _ = _exact_step(foam, load, start, dt)
            x.append(law.points + y[:, :3])
            v.append(2/dt*y)
            turn.append(_turn(y[:, 3:]))
        return dict(x=torch.cat(x), v=torch.cat(v), rotation=torch.cat(turn))
    if form == 'mixed' and case['nx']*case['ny']*case['nz'] > 300000:
        return None                                  # minutes of plain torch
    foam = _foam(case['nx'], case['ny'], case['nz'], seed, case['young'], case['contacts'])
    load = torch.as_tensor(_weight(foam), device=DEVICE)
    v = _velocity(foam, seed)
    if form in ('newton', 'mixed'):
        law, y, _ = _exact_step(foam, load, v, dt)
        out = dict(x=law.points + y[:, :3], v=2/dt*y - v, rotation=_turn(y[:, 3:]))
        if form == 'newton':
            n, _, fn, fs, mt, mb = law.trial(law.points, law.history, law.k, y, end=True)
            out.update(normal=n, fn=fn[:, 0], fs=fs, mt=mt[:, 0], mb=mb, work=float((load*y).sum()))
        return out
    if form == 'jacobian':
        law = _Law(foam)
        s = _Prestressed(law, float(law.radii.max()))
        _prestress(s, seed)
        history = (law.history[0], law.history[1], s.fn[:, None], s.fs, s.mt[:, None], s.mb)
        y, d = _displacement(foam, seed, 5e-3), _direction(foam, seed)
        return torch.func.jvp(lambda z: law.residual(law.points, v, history, law.k, load, dt, z), (y,), (d,))[1]
    if form == 'hvp':
        return _exact_hvp(foam, load, v, dt, seed)
    if form == 'linear':
        law = _Law(dict(foam, contacts=foam['contacts'] if foam['contacts'] is not None else
                        .5*(foam['points'][foam['pairs'][:, 0]] + foam['points'][foam['pairs'][:, 1]])))
        tangent = (law.history[0], law.contact - law.points[law.i], law.contact - law.points[law.j])
        rhs = dt*law.mass*v + .5*dt*dt*load
        rhs[law.fixed] = 0.
        dq = law.solver(tangent, law.k, dt)(rhs)
        return dict(q=dq, v=2/dt*dq - v, kq=law.stiffness(dq, tangent, law.k), work=float((load*dq).sum()))
    if form == 'energy':
        return _exact_energy(foam, seed)
    return _exact_adjoint(case, foam, load, v, seed)


class _Prestressed:
    """The names that _prestress reads and writes."""

    def __init__(self, law, radius):
        self.kn, self.ks, self.kb, self.kt = law.k.T
        self.normal, self.radii = law.history[0], law.radii


def _exact_hvp(foam, load, v, dt, seed):
    """(diag M + dt^2/4 K) q on the tangent that a step leaves behind: that of the
    committed end state, on which the next step starts."""
    law, y, _ = _exact_step(foam, load, v, dt)
    q = _direction(foam, seed).float().to(F64)
    x = law.points + y[:, :3]
    n, offset, *_ = law.trial(law.points, law.history, law.k, y, end=True)
    contact = law.geometry(x)[1] + offset
    out = law.mass*q + .25*dt*dt*law.stiffness(q, (n, contact - x[law.i], contact - x[law.j]), law.k)
    return torch.where(law.fixed[:, None], q, out)


def _exact_energy(foam, seed):
    contacts = foam['contacts']
    if contacts is None:
        contacts = .5*(foam['points'][foam['pairs'][:, 0]] + foam['points'][foam['pairs'][:, 1]])
    law = _Law(dict(foam, contacts=contacts))
    turn = _displacement(foam, seed, .05)
    theta = .1*_velocity(foam, seed + 5)[:, :4]/.02
    k = law.k*torch.exp(.5*(theta[law.i] + theta[law.j]))
    n0, ri, rj = law.history[0], law.contact - law.points[law.i], law.contact - law.points[law.j]

    rest = _turn(turn[:, 3:])
    x = (law.points + turn[:, :3]).requires_grad_(True)
    spin = torch.zeros_like(x, requires_grad=True)     # a further world rotation of every body, to first order
    frame = rest + torch.linalg.cross(spin[:, None, :], rest.transpose(1, 2), dim=2).transpose(1, 2)
    a, b = frame[law.i], frame[law.j]
    move = lambda matrix, r: (matrix@r[:, :, None])[:, :, 0]
    gap = x[law.j] + move(b, rj) - x[law.i] - move(a, ri)
    d = .5*(move(a.transpose(1, 2), gap) + move(b.transpose(1, 2), gap))
    psi = a.transpose(1, 2)@b
    skew = .5*(psi - psi.transpose(1, 2))
    phi = torch.stack((skew[:, 2, 1], skew[:, 0, 2], skew[:, 1, 0]), 1)
    dn, pn = _dot(d, n0), _dot(phi, n0)
    across, bend = d - dn*n0, phi - pn*n0
    energy = .5*(k*torch.cat((dn*dn, _dot(across, across), _dot(bend, bend), pn*pn), 1)).sum()
    return tuple(-g for g in torch.autograd.grad(energy, (x, spin)))


def _exact_adjoint(case, foam, load, v, seed):
    law, dt, steps = _Law(foam), case['dt'], case['steps']
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed) + 3)
    factor = torch.exp(.3*torch.randn(len(law.i), generator=gen, device=DEVICE, dtype=F64))
    k = (law.k*factor[:, None]).requires_grad_(True)
    loads = load[None].repeat(steps, 1, 1).requires_grad_(True)
    x0, v0 = law.points.clone().requires_grad_(True), v.clone().requires_grad_(True)
    ramp = torch.arange(steps + 1, device=DEVICE, dtype=F64)[:, None, None]/steps
    target = law.points + ramp*_displacement(foam, seed + 4, 1e-2)[:, :3]
    x, speed, history, positions = x0, v0, law.history, [x0]
    free = (~law.fixed)[:, None].to(F64)
    for t in range(steps):
        now = [a.detach() for a in (x, speed, k, loads[t])]
        past = tuple(a.detach() for a in history)
        y = law.increment(now[0], now[1], past, now[2], now[3], dt)
        y.requires_grad_(True)
        r = law.residual(now[0], now[1], past, now[2], now[3], dt, y)
        solve = law.solver(law.trial(now[0], past, now[2], y.detach())[1], now[2], dt, 1e-8)

        def transposed(g, r=r, y=y, solve=solve):
            g = g*free
            lam = torch.zeros_like(g)
            for _ in range(40):
                change = solve(g - torch.autograd.grad(r, y, lam, retain_graph=True)[0]*free)
                lam = lam + change
                if bool((change*change).sum() <= 1e-30*(lam*lam).sum()):
                    break
            return lam
        y = y.detach() + _Implicit.apply(law.residual(x, speed, history, k, loads[t], dt, y.detach()), transposed)
        history = law.trial(x, history, k, y, end=True)
        x, speed = x + y[:, :3], 2/dt*y - speed
        positions.append(x)
    positions = torch.stack(positions)
    grads = torch.autograd.grad(((positions - target)**2).sum(), (k, loads, x0, v0))
    return dict(positions=positions.detach(), stiffness=grads[0], loads=grads[1], x=grads[2], v=grads[3])
