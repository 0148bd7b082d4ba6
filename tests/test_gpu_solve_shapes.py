"""Every plane shape of the Fourier solves against the three-dimensional cuFFT
path, with the density painted per cell (two cells per particle and axis) and
as z pairs (one): the row and column transforms are instantiated per side, so
each pair of sides is its own kernel."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def fpm(cuda):
  import flowpm_b200
  return flowpm_b200


def _forces(dims, flags, disp):
  from flowpm_b200 import _lib
  from flowpm_b200._plans import Plan
  plan = Plan(dims, flags=flags)
  try:
    f = torch.empty_like(disp)
    _lib.call('fpm_force', plan.handle, _lib.ptr(disp),
              _lib.dvec([0.45] * len(dims)), _lib.ptr(f), _lib.stream_ptr())
    torch.cuda.synchronize()
    return f
  finally:
    plan.close()


# (nx, ny, nz) of the force mesh; 256 and 512 along y and z take the row and
# column passes of meshes that one block cannot hold
MESHES = ([(16, ny, nz) for ny in (16, 32, 64, 128)
           for nz in (16, 32, 64, 128)] +
          [(32, 16, 32), (64, 32, 16), (128, 16, 64)] +
          [(256, ny, nz) for ny in (256, 512) for nz in (256, 512)] +
          [(512, 256, 256)])


@pytest.mark.parametrize('mesh', MESHES, ids=lambda m: '%dx%dx%d' % m)
@pytest.mark.parametrize('bf', [1, 2])
def test_solve_shape(fpm, mesh, bf):
  from flowpm_b200 import _lib
  nx, ny, nz = (n // bf for n in mesh)
  count = 2 if nx * ny * nz < 1 << 20 else 1
  dims = [(nx, ny, nz, bf)] * count
  g = torch.Generator(device='cuda').manual_seed(3)
  disp = torch.randn((count * nx * ny * nz, 3), generator=g,
                     device='cuda') * 1.5
  f = _forces(dims, 0, disp)
  r = _forces(dims, _lib.FPM_PLAN_CUFFT, disp)
  # both transforms round at 6e-8 per stage: log2(cells) < 28 stages each way
  err = rel_l2(f.cpu().numpy(), r.cpu().numpy())
  assert err < 2 * 28 * 6e-8 * 3, err
