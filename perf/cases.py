"""The work whose speed is watched: simulations, gradients, batches and mesh
analysis as a program that uses ``flowpm_b200`` calls them.

``listed()`` are the named cases, ``draw(rng)`` gives more of the same kinds
and ranges, ``prepare`` makes what a program holds before the call, ``run`` is
one pass through the public API, ``work`` the bytes and operations the pass
cannot do without, and ``exact`` the same outputs in 64 bits, in plain torch.

Kinds of case:

* ``nbody``: a particle-mesh simulation from a given initial state;
* ``grad``: density of a simulation from its linear field, and the gradient
  of a chi^2 with respect to that field (initial-condition reconstruction);
* ``many``: simulations of uneven size and step count in one batch;
* ``lpt``: 1LPT / 2LPT initial conditions from a linear field;
* ``cic``: paint of a particle catalogue, readout at its particles, and
  (``grad``) their gradients;
* ``power``: binned power spectrum of a field;
* ``planes``: lensing density planes of a snapshot, and (``grad``) the
  gradient with respect to its positions.
"""
import math

import numpy as np
import torch

import flowpm_b200 as fpm

# Planck 2015 (flowpm/cosmology.py Planck15)
_COSMO = dict(Omega_c=0.2589, Omega_b=0.0486, h=0.6774, n_s=0.9667,
              sigma8=0.8159, Omega_k=0.0, w0=-1.0, wa=0.0)
_OM = _COSMO['Omega_c'] + _COSMO['Omega_b']
_A0 = 0.1  # scale factor of the initial conditions


def listed():
  return [
      # the smallest call: one toy box, where launches and host work count
      dict(name='nbody_32', kind='nbody', nx=32, ny=32, nz=32, batch=1, bf=1,
           steps=10, box=100.0),
      # the benchmark's simulation: 128^3 in 200 Mpc/h, 40 KDK steps
      dict(name='nbody_128', kind='nbody', nx=128, ny=128, nz=128, batch=1,
           bf=1, steps=40, box=200.0),
      # force mesh twice as fine as the particles (pm_nc_factor = 2)
      dict(name='nbody_fine_mesh', kind='nbody', nx=128, ny=128, nz=128,
           batch=1, bf=2, steps=10, box=400.0),
      # a batch on a mesh without a power of two, unequal axes
      dict(name='nbody_odd', kind='nbody', nx=90, ny=100, nz=126, batch=2,
           bf=1, steps=10, box=300.0),
      # the largest box of the benchmark, a few steps of it
      dict(name='nbody_512', kind='nbody', nx=512, ny=512, nz=512, batch=1,
           bf=1, steps=5, box=1000.0),
      # reconstruction: gradients of two small boxes at once
      dict(name='grad_64', kind='grad', nx=64, ny=64, nz=64, batch=2, bf=1,
           steps=10, box=100.0, order=2),
      # reconstruction at the benchmark's size: 128^3, 20 steps
      dict(name='grad_128', kind='grad', nx=128, ny=128, nz=128, batch=1,
           bf=1, steps=20, box=200.0, order=2),
      # an emulator's training set: uneven simulations in one batch
      dict(name='many', kind='many', n32=8, n64=4, n128=2, steps=10,
           box=200.0),
      # 2LPT initial conditions (mock catalogues)
      dict(name='lpt_256', kind='lpt', nx=256, ny=256, nz=256, batch=1,
           box=500.0, order=2),
      # a weighted catalogue in no order painted and read back, with gradients
      dict(name='cic_catalogue', kind='cic', nx=200, ny=180, nz=150, batch=1,
           npart=2000003, weighted=True, grad=True),
      # power spectrum of one large field
      dict(name='power_256', kind='power', nx=256, ny=256, nz=256, batch=1,
           box=500.0, kmin=0.0123, dk=0.0117),
      # lensing planes of a snapshot, with the gradient for its positions
      dict(name='planes', kind='planes', nx=128, ny=128, nz=128, batch=1,
           nplanes=8, res=512, rotate=True, grad=True),
  ]


def _between(rng, lo, hi):
  """A whole number in [lo, hi], spread over its logarithm."""
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, lo, hi):
  """Mesh sides: a cube of a usual size, or unequal sides, odd ones among
  them (z even or odd)."""
  usual = [n for n in (16, 24, 32, 48, 64, 96, 100, 128, 160, 192, 200, 256)
           if lo <= n <= hi]
  if rng.random() < 0.6:
    n = rng.choice(usual)
    return n, n, n
  return tuple(_between(rng, lo, hi) for _ in range(3))


def draw(rng):
  kind = rng.choice(['nbody', 'nbody', 'nbody', 'grad', 'grad', 'many', 'lpt',
                     'cic', 'power', 'planes'])
  if kind == 'nbody':
    nx, ny, nz = _mesh(rng, 16, 256)
    np_ = nx * ny * nz
    bf = 2 if np_ <= 128**3 and rng.random() < 0.3 else 1
    batch = rng.choice([1, 1, 2, 4]) if np_ <= 128**3 else 1
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, batch=batch, bf=bf,
                steps=_between(rng, 1, 20 if np_ <= 128**3 else 5),
                box=nx * rng.uniform(1.0, 4.0))
  if kind == 'grad':
    nx, ny, nz = _mesh(rng, 16, 128)
    batch = rng.choice([1, 2, 4]) if nx * ny * nz <= 64**3 else 1
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, batch=batch,
                bf=2 if nx * ny * nz <= 64**3 and rng.random() < 0.3 else 1,
                steps=_between(rng, 1, 12), box=nx * rng.uniform(1.5, 4.0),
                order=rng.choice([1, 2]))
  if kind == 'many':
    return dict(kind=kind, n32=rng.randint(1, 12), n64=rng.randint(1, 6),
                n128=rng.randint(0, 2), steps=_between(rng, 3, 16),
                box=rng.uniform(100.0, 400.0))
  if kind == 'lpt':
    nx, ny, nz = _mesh(rng, 16, 256)
    batch = rng.choice([1, 2]) if nx * ny * nz <= 128**3 else 1
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, batch=batch,
                box=nx * rng.uniform(1.0, 4.0), order=rng.choice([1, 2]))
  if kind == 'cic':
    nx, ny, nz = _mesh(rng, 16, 256)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, batch=rng.choice([1, 2]),
                npart=_between(rng, 1000, 4000000),
                weighted=rng.random() < 0.5, grad=rng.random() < 0.5)
  if kind == 'power':
    nx, ny, nz = _mesh(rng, 16, 256)
    box = nx * rng.uniform(1.0, 4.0)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, batch=rng.choice([1, 2]),
                box=box, kmin=2 * math.pi / box * rng.uniform(0.9, 1.1),
                dk=2 * math.pi / box * rng.uniform(0.8, 2.5))
  nx, ny, nz = _mesh(rng, 32, 160)
  return dict(kind=kind, nx=nx, ny=ny, nz=nz, batch=1,
              nplanes=rng.randint(1, 16), res=_between(rng, 64, 1024),
              rotate=rng.random() < 0.5, grad=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed):
  return torch.Generator(device='cuda').manual_seed(int(seed) * 7919 + 17)


def _freq(n, half=False):
  f = torch.fft.rfftfreq(n, device='cuda', dtype=torch.float64) if half else \
      torch.fft.fftfreq(n, device='cuda', dtype=torch.float64)
  return 2 * math.pi * f


def _bbks(k):
  """Shape of the linear power spectrum: k T(k)^2 (Bardeen et al. 1986)."""
  q = k / 0.21
  t = torch.log1p(2.34 * q) / (2.34 * q) * (
      1 + 3.89 * q + (16.1 * q)**2 + (5.46 * q)**3 + (6.71 * q)**4)**-0.25
  return k * t * t


def _amplitude():
  """Normalisation of _bbks to sigma8."""
  k = torch.logspace(-4, 2, 8192, dtype=torch.float64)
  x = 8.0 * k
  w = 3 * (torch.sin(x) - x * torch.cos(x)) / x**3
  y = _bbks(k) * w * w * k**3 / (2 * math.pi**2)
  var = float(torch.trapezoid(y, torch.log(k)))
  return _COSMO['sigma8']**2 / var


def _linear_modes(nc, batch, box, gen):
  """Half spectrum of a Gaussian linear field (overdensity at a = 1) on
  cells of box / nx, and k^2 in cell units."""
  nx, ny, nz = nc
  h = box / nx
  white = torch.randn((batch, nx, ny, nz), generator=gen, device='cuda')
  fk = torch.fft.rfftn(white, dim=(1, 2, 3))
  del white
  k2 = (_freq(nx)[:, None, None]**2 + _freq(ny)[None, :, None]**2 +
        _freq(nz, True)[None, None, :]**2)
  k2[0, 0, 0] = 1.0
  amp = torch.sqrt(_amplitude() * _bbks(torch.sqrt(k2) / h) / h**3)
  amp[0, 0, 0] = 0.0
  return fk * amp.float(), k2.float()


def _linear(nc, batch, box, gen):
  fk, _ = _linear_modes(nc, batch, box, gen)
  return torch.fft.irfftn(fk, s=tuple(nc), dim=(1, 2, 3)).contiguous()


def _lattice(nc, dtype=torch.float32):
  ax = [torch.arange(n, device='cuda', dtype=dtype) for n in nc]
  return torch.stack(torch.meshgrid(*ax, indexing='ij'), -1).reshape(-1, 3)


def _initial_state(nc, batch, box, gen, growth=0.128):
  """Zel'dovich state (3, batch, npart, 3) at a = 0.1 (growth the linear
  growth factor there)."""
  fk, k2 = _linear_modes(nc, batch, box, gen)
  fk = fk / k2
  del k2
  state = torch.empty((3, batch, nc[0] * nc[1] * nc[2], 3), device='cuda')
  for d in range(3):
    k = _freq(nc[d], d == 2).float()
    if nc[d] % 2 == 0:
      k[nc[d] // 2] = 0.0
    shape = [1, 1, 1, 1]
    shape[d + 1] = -1
    psi = torch.fft.irfftn(fk * (1j * k.reshape(shape)), s=tuple(nc),
                           dim=(1, 2, 3))
    state[0, ..., d] = growth * psi.reshape(batch, -1)
  state[1] = 0.175 * state[0]  # a^2 f1 E at a = 0.1
  state[2] = 0.26 * state[0]
  state[0] += _lattice(nc)
  return state


def _stages(steps):
  return np.linspace(_A0, 1.0, steps + 1)


def _many_sims(case):
  """(nc, steps, box) of each simulation of a ``many`` case."""
  out = []
  for n, count in ((32, case['n32']), (64, case['n64']), (128, case['n128'])):
    for i in range(count):
      out.append((n, max(1, case['steps'] - i), case['box'] * n / 128))
  return out


def _rotation():
  c, s = math.cos(0.3), math.sin(0.3)
  rz = np.array([[c, -s, 0], [s, c, 0], [0, 0, 1.0]])
  rx = np.array([[1.0, 0, 0], [0, c, -s], [0, s, c]])
  return rx @ rz


def prepare(case, seed):
  gen = _gen(seed)
  kind = case['kind']
  s = dict(case=case)
  if kind == 'many':
    sims = _many_sims(case)
    s['cosmo'] = fpm.cosmology.Cosmology(**_COSMO)
    s['states'] = [_initial_state([n] * 3, 1, box, gen)
                   for n, _, box in sims]
    s['runner'] = fpm.BatchRunner([
        dict(nc=n, cosmo=s['cosmo'], stages=_stages(t)) for n, t, _ in sims])
    return s
  nc = [case['nx'], case['ny'], case['nz']]
  s['nc'] = nc
  if kind == 'cic':
    size = torch.tensor(nc, dtype=torch.float32, device='cuda')
    B, n = case['batch'], case['npart']
    # half of the particles uniform, half in clumps of about two cells
    x = torch.rand((B, n, 3), generator=gen, device='cuda') * size
    m = n // 2
    centre = torch.rand((B, 256, 3), generator=gen, device='cuda') * size
    which = torch.randint(256, (m,), generator=gen, device='cuda')
    x[:, :m] = centre[:, which] + 2.0 * torch.randn(
        (B, m, 3), generator=gen, device='cuda')
    x = x[:, torch.randperm(n, generator=gen, device='cuda')].contiguous()
    s['part'] = x
    s['weight'] = (0.5 + torch.rand((B, n), generator=gen, device='cuda')
                   if case['weighted'] else None)
    s['mesh'] = torch.zeros([B] + nc, device='cuda')
    s['g_mesh'] = torch.randn([B] + nc, generator=gen, device='cuda')
    s['g_read'] = torch.randn((B, n), generator=gen, device='cuda')
    for k in ('part', 'weight', 'mesh'):
      if case['grad'] and s[k] is not None:
        s[k].requires_grad_(True)
    return s
  if kind == 'planes':
    s['state'] = _initial_state(nc, case['batch'], 2.0 * nc[0], gen,
                                growth=0.7)
    edges = np.linspace(0.0, nc[2], case['nplanes'] + 1)
    s['centers'] = 0.5 * (edges[1:] + edges[:-1])
    s['width'] = float(edges[1])
    s['rotation'] = _rotation() if case['rotate'] else None
    s['shift'] = [0.11, 0.23, 0.07] if case['rotate'] else None
    if case['grad']:
      s['state'].requires_grad_(True)
      s['g'] = torch.randn((case['batch'], case['nplanes'], case['res'],
                            case['res']), generator=gen, device='cuda')
    return s
  if kind == 'power':
    s['field'] = _linear(nc, case['batch'], case['box'], gen)
    return s
  s['cosmo'] = fpm.cosmology.Cosmology(**_COSMO)
  if kind == 'nbody':
    s['stages'] = _stages(case['steps'])
    s['state'] = _initial_state(nc, case['batch'], case['box'], gen)
  elif kind == 'lpt':
    s['linear'] = _linear(nc, case['batch'], case['box'], gen)
  else:  # grad
    s['stages'] = _stages(case['steps'])
    s['linear'] = _linear(nc, case['batch'], case['box'],
                          gen).requires_grad_(True)
    s['mesh'] = torch.zeros([case['batch']] + nc, device='cuda')
    s['data'] = 1.0 + _linear(nc, case['batch'], case['box'], gen)
  return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
  case = s['case']
  kind = case['kind']
  if kind == 'nbody':
    return fpm.nbody(s['cosmo'], s['state'], s['stages'], s['nc'],
                     pm_nc_factor=case['bf'])
  if kind == 'grad':
    state = fpm.lpt_init(s['cosmo'], s['linear'], _A0, order=case['order'])
    state = fpm.nbody(s['cosmo'], state, s['stages'], s['nc'],
                      pm_nc_factor=case['bf'])
    rho = fpm.cic_paint(s['mesh'], state[0])
    loss = 0.5 * torch.sum((rho - s['data'])**2)
    grad, = torch.autograd.grad(loss, s['linear'])
    return dict(density=rho.detach(), gradient=grad)
  if kind == 'many':
    s['runner'].load(s['states'])
    s['runner'].run()
    return s['runner'].results()
  if kind == 'lpt':
    return fpm.lpt_init(s['cosmo'], s['linear'], _A0, order=case['order'])
  if kind == 'power':
    k, p = fpm.power_spectrum(s['field'], kmin=case['kmin'], dk=case['dk'],
                              boxsize=[case['box']] * 3)
    return dict(k=k, power=p)
  if kind == 'cic':
    mesh = fpm.cic_paint(s['mesh'], s['part'], weight=s['weight'])
    read = fpm.cic_readout(mesh, s['part'])
    if not case['grad']:
      return dict(mesh=mesh, read=read)
    wrt = [t for t in (s['mesh'], s['part'], s['weight']) if t is not None]
    grads = torch.autograd.grad([mesh, read], wrt,
                                [s['g_mesh'], s['g_read']])
    return dict(mesh=mesh.detach(), read=read.detach(), grads=list(grads))
  planes = fpm.raytracing.density_planes(
      s['state'], s['nc'], s['centers'], s['width'], case['res'],
      rotation=s['rotation'], shift=s['shift'])
  if not case['grad']:
    return planes
  grad, = torch.autograd.grad(planes, s['state'], s['g'])
  return dict(planes=planes.detach(), grad=grad[0])


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _force_work(np_, cells):
  """Bytes and operations of one leapfrog step: the particles read and
  written once (d, p), the density written once and read once, the three
  force meshes written once and read once, each with the spectrum's round
  trip through a transform pass; the FFT pair, paint and readout."""
  bytes_ = 48 * np_ + 8 * cells + 24 * cells + 32 * cells
  flops = 2 * 2.5 * cells * math.log2(max(2, cells)) + 24 * cells + 150 * np_
  return bytes_, flops


def work(case):
  kind = case['kind']
  if kind == 'many':
    b = f = 0
    for n, t, _ in _many_sims(case):
      db, df = _force_work(n**3, n**3)
      b += (t + 1) * db + 60 * n**3
      f += (t + 1) * df
    return dict(bytes=b, flops=f)
  np_ = case['nx'] * case['ny'] * case['nz'] * case['batch']
  fft = 2.5 * np_ * math.log2(np_)
  if kind == 'nbody':
    b, f = _force_work(np_, np_ * case['bf']**3)
    n = case['steps'] + 1
    return dict(bytes=n * b + 60 * np_, flops=n * f)
  if kind == 'grad':
    b, f = _force_work(np_, np_ * case['bf']**3)
    n = case['steps'] + 1
    return dict(bytes=3 * n * b + 200 * np_, flops=3 * n * f + 20 * fft)
  if kind == 'lpt':
    second = case['order'] == 2
    return dict(bytes=40 * np_ + (48 if second else 0) * np_,
                flops=(14 if second else 4) * fft)
  if kind == 'power':
    return dict(bytes=4 * np_ + 8 * np_, flops=fft + 10 * np_)
  if kind == 'cic':
    n = case['npart'] * case['batch']
    per = 12 + 4 + (4 if case['weighted'] else 0)
    if case['grad']:
      return dict(bytes=n * (2 * per + 12 + 8) + 20 * np_, flops=300 * n)
    return dict(bytes=n * per + 12 * np_, flops=100 * n)
  cells = case['nplanes'] * case['res']**2 * case['batch']
  if case['grad']:
    return dict(bytes=(24 + 36) * np_ + 8 * cells, flops=120 * np_)
  return dict(bytes=12 * np_ + 4 * cells, flops=60 * np_)


# ---------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _hubble(a):
  return np.sqrt(_OM / a**3 + (1 - _OM))


def _rhs(a, y):
  e2 = _OM / a**3 + (1 - _OM)
  om, ode = _OM / a**3 / e2, (1 - _OM) / e2
  fric = (ode - 0.5 * om + 2.0) / a
  return np.stack([y[1], 1.5 * om * y[0] / a**2 - fric * y[1],
                   y[3], 1.5 * om * (y[2] - y[0]**2) / a**2 - fric * y[3]])


_TABLE = []


def _growth_table():
  """Growth factors D1, D1', D2, D2' and their derivatives on the model's
  grid: 256 scale factors from 0.01 to 1, fourth-order Runge-Kutta."""
  if not _TABLE:
    a = np.logspace(-2, 0, 256)
    y = np.array([a[0], 1.0, -3 / 7 * a[0]**2, -6 / 7 * a[0]])
    rows = [y]
    for t, u in zip(a[:-1], a[1:]):
      dt = u - t
      k1 = _rhs(t, y)
      k2 = _rhs(t + dt / 2, y + dt / 2 * k1)
      k3 = _rhs(t + dt / 2, y + dt / 2 * k2)
      k4 = _rhs(t + dt, y + dt * k3)
      y = y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
      rows.append(y)
    y = np.stack(rows, 1)
    d = _rhs(a, y)
    one, two = y[0, -1], y[2, -1]
    _TABLE.append((np.log(a), dict(
        D1=y[0] / one, D1f=y[1] / one, F1=d[1] / one,
        D2=y[2] / two, D2f=y[3] / two, F2=d[3] / two)))
  return _TABLE[0]


def _of(name, a):
  x, t = _growth_table()
  return float(np.interp(np.log(a), x, t[name]))


def _G(a, n=1):
  return _of('D%df' % n, a) * a**3 * _hubble(a)


def _dG(a, n=1):
  e = _hubble(a)
  de = -1.5 * _OM / a**4 / e
  d = _of('D%df' % n, a)
  return _of('F%d' % n, a) * a**3 * e + d * a**3 * de + 3 * a**2 * e * d


def _kick(ai, ac, af):
  return (_G(af) - _G(ai)) / (ac**2 * _hubble(ac) * _dG(ac))


def _drift(ai, ac, af):
  return (_of('D1', af) - _of('D1', ai)) / (
      ac**3 * _hubble(ac) * _of('D1f', ac))


def _corners(x, nc):
  """Weight and cell of the 8 neighbours of positions x (npart, 3)."""
  lo = torch.floor(x.detach())
  for c in range(8):
    nb = lo + torch.tensor([c & 1, (c >> 1) & 1, c >> 2], device='cuda',
                           dtype=torch.float64)
    w = (1 - (x - nb).abs()).prod(-1)
    i = nb.long()
    yield w, ((i[:, 0] % nc[0]) * nc[1] + i[:, 1] % nc[1]) * nc[2] + \
        i[:, 2] % nc[2]


def _paint64(mesh, x, weight=None):
  out = mesh.reshape(-1)
  for w, cell in _corners(x, mesh.shape):
    out = out.index_add(0, cell, w if weight is None else weight * w)
  return out.reshape(mesh.shape)


def _read64(meshes, x):
  out = [0.0] * len(meshes)
  for w, cell in _corners(x, meshes[0].shape):
    for d, m in enumerate(meshes):
      out[d] = out[d] + m.reshape(-1)[cell] * w
  return torch.stack(out, -1)


def _k2(nc):
  k2 = (_freq(nc[0])[:, None, None]**2 + _freq(nc[1])[None, :, None]**2 +
        _freq(nc[2], True)[None, None, :]**2)
  k2[0, 0, 0] = 1.0
  return k2


def _ik(nc, d):
  """The four-point gradient along axis d."""
  k = _freq(nc[d], d == 2)
  g = (8 * torch.sin(k) - torch.sin(2 * k)) / 6
  shape = [1, 1, 1]
  shape[d] = -1
  return 1j * g.reshape(shape)


def _force64(x, nc, bf):
  """Force of one simulation at positions x (npart, 3) in lattice units."""
  nm = [n * bf for n in nc]
  y = x * bf
  rho = _paint64(torch.zeros(nm, device='cuda', dtype=torch.float64), y)
  pot = torch.fft.rfftn(rho * bf**3) / _k2(nm)
  del rho
  f = _read64([torch.fft.irfftn(pot * _ik(nm, d), s=nm) for d in range(3)], y)
  return f * (1.5 * _OM / bf)


def _nbody64(x, p, nc, bf, stages, keep=True):
  """Positions, momenta and forces of one simulation; with keep False every
  step is recomputed in the backward instead of kept."""
  from torch.utils.checkpoint import checkpoint

  def step(x, p, f, a0, a1):
    ah = (a0 * a1)**0.5
    p = p + _kick(a0, a0, ah) * f
    x = x + _drift(a0, ah, a1) * p
    f = _force64(x, nc, bf)
    return x, p + _kick(ah, a1, a1) * f, f

  f = _force64(x, nc, bf) if keep else checkpoint(
      lambda q: _force64(q, nc, bf), x, use_reentrant=False)
  for a0, a1 in zip(stages[:-1], stages[1:]):
    a0, a1 = float(a0), float(a1)
    if keep:
      x, p, f = step(x, p, f, a0, a1)
    else:
      x, p, f = checkpoint(step, x, p, f, a0, a1, use_reentrant=False)
  return x, p, f


def _lpt64(linear, order):
  """2LPT state (3, npart, 3) at a = 0.1 of one linear field."""
  nc = list(linear.shape)
  a, e = _A0, _hubble(_A0)
  psi = lambda fk: torch.stack([  # noqa: E731
      torch.fft.irfftn(fk / _k2(nc) * _ik(nc, d), s=nc).reshape(-1)
      for d in range(3)], -1)
  fk = torch.fft.rfftn(linear)
  x1 = _of('D1', a) * psi(fk)
  state = [x1, a**2 * e * (a * _of('D1f', a) / _of('D1', a)) * x1,
           a**2 * e * _dG(a) / _of('D1', a) * x1]
  if order == 2:
    hess = lambda i, j: torch.fft.irfftn(  # noqa: E731
        fk / _k2(nc) * _ik(nc, i) * _ik(nc, j), s=nc)
    h = [hess(d, d) for d in range(3)]
    src = h[1] * h[2] + h[2] * h[0] + h[0] * h[1]
    for i, j in ((1, 2), (2, 0), (0, 1)):
      src = src - hess(i, j)**2
    x2 = _of('D2', a) * psi(torch.fft.rfftn(src * (3.0 / 7.0)))
    state = [state[0] + x2,
             state[1] + a**2 * e * (a * _of('D2f', a) / _of('D2', a)) * x2,
             state[2] + a**2 * e * _dG(a, 2) / _of('D2', a) * x2]
  return torch.stack([state[0] + _lattice(nc, torch.float64)] + state[1:])


def _power64(field, case):
  n, box = list(field.shape[1:]), case['box']
  kmax = np.pi * min(n) / box + case['dk'] / 2
  edges = np.arange(case['kmin'], kmax, case['dk'])
  k = torch.sqrt(sum((_freq(m).reshape([-1 if i == d else 1 for i in range(3)])
                      * (m / box))**2 for d, m in enumerate(n)))
  which = torch.bucketize(k.reshape(-1), torch.tensor(edges, device='cuda'),
                          right=True)
  w = torch.full(n, 2.0, device='cuda', dtype=torch.float64)
  w[..., 0] = 1.0
  w[..., -1] = 1.0
  w = w.reshape(-1)
  out = []
  for f in field:
    p = torch.fft.fftn(f.double()).abs().square().reshape(-1)
    tot = torch.bincount(which, weights=w * p, minlength=len(edges) + 1)
    cnt = torch.bincount(which, weights=w, minlength=len(edges) + 1)
    out.append((tot / cnt)[1:-1] * box**3 / float(np.prod(n))**2)
  return dict(k=edges[:-1] + (edges[1:] - edges[:-1]) / 2,
              power=torch.stack(out))


def _planes64(x, s):
  """Density planes of positions x (npart, 3)."""
  case, nc = s['case'], s['nc']
  res = case['res']
  if s['rotation'] is not None:
    x = x @ torch.tensor(s['rotation'], device='cuda').T
    x = x + torch.tensor(np.array(nc) * s['shift'], device='cuda')
  u = torch.remainder(x[:, :2], nc[0]) / nc[0] * res
  out = []
  for c in s['centers']:
    inside = ((x[:, 2] > c - s['width'] / 2) &
              (x[:, 2] <= c + s['width'] / 2)).double()
    plane = torch.zeros(res * res, device='cuda', dtype=torch.float64)
    lo = torch.floor(u.detach())
    for q in range(4):
      nb = lo + torch.tensor([q & 1, q >> 1], device='cuda',
                             dtype=torch.float64)
      i = nb.long() % res
      plane = plane.index_add(0, i[:, 0] * res + i[:, 1],
                              (1 - (u - nb).abs()).prod(-1) * inside)
    out.append(plane.reshape(res, res) /
               ((nc[0] / res) * (nc[1] / res) * s['width']))
  return torch.stack(out)


def exact(case, seed):
  kind = case['kind']
  s = prepare(case, seed)
  if kind == 'many':
    s['runner'].close()
    with torch.no_grad():
      return [torch.stack(_nbody64(
          st[0, 0].double(), st[1, 0].double(), [n] * 3, 1,
          _stages(t)))[:, None]
              for st, (n, t, _) in zip(s['states'], _many_sims(case))]
  nc = s['nc']
  if kind == 'nbody':
    with torch.no_grad():
      out = [torch.stack(_nbody64(
          s['state'][0, b].double(), s['state'][1, b].double(), nc,
          case['bf'], s['stages'])) for b in range(case['batch'])]
    return torch.stack(out, 1)
  if kind == 'lpt':
    return torch.stack([_lpt64(f.double(), case['order'])
                        for f in s['linear']], 1)
  if kind == 'grad':
    rho, grad = [], []
    for b in range(case['batch']):
      lin = s['linear'][b].detach().double().requires_grad_(True)
      x, p, _ = _lpt64(lin, case['order'])
      x = _nbody64(x, p, nc, case['bf'], s['stages'], keep=False)[0]
      r = _paint64(s['mesh'][b].double(), x)
      loss = 0.5 * torch.sum((r - s['data'][b].double())**2)
      grad.append(torch.autograd.grad(loss, lin)[0])
      rho.append(r.detach())
    return dict(density=torch.stack(rho), gradient=torch.stack(grad))
  if kind == 'power':
    return _power64(s['field'], case)
  if kind == 'cic':
    meshes, reads, grads = [], [], []
    for b in range(case['batch']):
      leaf = [s[k][b].detach().double().requires_grad_(case['grad'])
              for k in ('mesh', 'part', 'weight') if s[k] is not None]
      m = _paint64(leaf[0], leaf[1], leaf[2] if len(leaf) > 2 else None)
      r = _read64([m], leaf[1])[:, 0]
      if case['grad']:
        grads.append(torch.autograd.grad(
            [m, r], leaf, [s['g_mesh'][b].double(), s['g_read'][b].double()]))
      meshes.append(m.detach())
      reads.append(r.detach())
    out = dict(mesh=torch.stack(meshes), read=torch.stack(reads))
    if case['grad']:
      out['grads'] = [torch.stack(g) for g in zip(*grads)]
    return out
  planes, grads = [], []
  for b in range(case['batch']):
    x = s['state'][0, b].detach().double().requires_grad_(case['grad'])
    p = _planes64(x, s)
    if case['grad']:
      grads.append(torch.autograd.grad(p, x, s['g'][b].double())[0])
    planes.append(p.detach())
  if not case['grad']:
    return torch.stack(planes)
  return dict(planes=torch.stack(planes), grad=torch.stack(grads))
