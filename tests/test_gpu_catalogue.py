"""CIC operators on catalogues and the lattice shift where the z neighbours of
a row change form: every place of a row in a 16-byte group, the wrap, meshes
that begin and end inside a group, and rows of one to five cells."""
import numpy as np
import pytest
import torch

from oracle import pm as opm

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def call(cuda):
  from flowpm_b200 import _lib

  def f(name, *args):
    _lib.call(name, *[_lib.ptr(a) if torch.is_tensor(a) or a is None else a
                      for a in args], _lib.stream_ptr())
  return f


def _at(a, offset):
  """a on the device, ``offset`` floats past a 16-byte boundary."""
  buf = torch.empty(a.size + 4, dtype=torch.float32, device='cuda')
  v = buf[offset:offset + a.size].view(a.shape)
  v.copy_(torch.tensor(a))
  return v


# Weights are products of three factors in [0, 1] with errors below 2e-7
# each, and a cell sums at most a few dozen of them: 1e-5 of the largest value
@pytest.mark.parametrize('shape,npart', [
    ((3, 4, 1), 60), ((2, 3, 2), 60), ((4, 2, 3), 60), ((3, 3, 4), 60),
    ((2, 2, 5), 60), ((5, 6, 16), 1500), ((4, 6, 34), 1500),
    ((1, 1, 31), 100), ((4, 4, 4), 1)])
@pytest.mark.parametrize('offset', [0, 1, 2, 3])
@pytest.mark.parametrize('weighted', [False, True])
def test_cic_catalogue(call, shape, npart, offset, weighted):
  B, rng = 2, np.random.default_rng(3 + offset)
  part = (rng.random((B, npart, 3)) * shape).astype(np.float32)
  # rows' last cells, and positions outside the box on both sides
  part[:, ::7, 2] = np.float32(shape[2] - 0.25)
  part[:, ::11] -= np.array(shape, np.float32)
  part[:, ::13] += np.array(shape, np.float32)
  w = rng.standard_normal((B, npart)).astype(np.float32) if weighted else None
  mesh = rng.standard_normal((B,) + shape).astype(np.float32)
  lout = rng.standard_normal((B, npart)).astype(np.float32)

  d = lambda a: None if a is None else torch.tensor(a, dtype=torch.float64,
                                                    requires_grad=True)
  xo, wo, mo = d(part), d(w), d(mesh)
  painted = opm.cic_paint(torch.zeros((B,) + shape, dtype=torch.float64), xo,
                          wo)
  gp = torch.autograd.grad((painted * mo.detach()).sum(),
                           [xo] + ([wo] if weighted else []))
  read = opm.cic_readout(mo, xo)
  gr = torch.autograd.grad((read * d(lout).detach()).sum(), [mo, xo])

  g = lambda a: None if a is None else torch.tensor(a, device='cuda')
  x, m, wd, lo = g(part), _at(mesh, offset), g(w), g(lout)
  dims = [B] + list(shape)
  acc = _at(mesh, offset)
  call('fpm_cic_paint', acc, *dims, x, npart, wd)
  out = torch.empty_like(lo)
  call('fpm_cic_readout', m, *dims, x, npart, out)
  lp, lw = torch.empty_like(x), torch.empty_like(lo)
  call('fpm_cic_paint_adjoint', m, *dims, x, npart, wd, lp, lw)
  lm, lx = _at(np.zeros_like(mesh), offset), torch.empty_like(x)
  call('fpm_cic_readout_adjoint', m, *dims, x, npart, lo, lm, lx)

  def check(a, b):
    a, b = a.cpu().numpy().astype(np.float64), b.detach().numpy()
    np.testing.assert_allclose(a, b.reshape(a.shape), rtol=0,
                               atol=1e-5 * max(1., np.abs(b).max()))

  check(acc, painted + mo)
  check(out, read)
  check(lp, gp[0])
  if weighted:
    check(lw, gp[1])
  check(lm, gr[0])
  check(lx, gr[1])


@pytest.mark.parametrize('shape', [(2, 3, 4), (3, 5, 8), (2, 3, 6), (3, 2, 1),
                                   (1, 1, 4), (7, 33, 12)])
@pytest.mark.parametrize('offset', [0, 1])
@pytest.mark.parametrize('sign', [1, -1])
def test_lattice_shift(call, shape, offset, sign):
  a = np.random.default_rng(5).standard_normal(
      (2,) + shape + (3,)).astype(np.float32)
  x, out = _at(a, offset), _at(a, 0)
  call('fpm_lattice_shift', x, out, 2, *shape, sign)
  q = np.stack(np.indices(shape), -1).astype(np.float32)
  # one rounded sum per component on both sides
  np.testing.assert_array_equal(out.cpu().numpy(), a + np.float32(sign) * q)
