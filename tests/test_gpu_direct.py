"""nbody working in its output (large runs) against its working buffers."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nc,batch,bf', [(16, 1, 1), (16, 3, 2), (20, 2, 1),
                                         (9, 1, 2)])
@pytest.mark.parametrize('steps', [0, 1, 4])
@pytest.mark.parametrize('pgd', [False, True])
def test_direct_nbody(cuda, monkeypatch, nc, batch, bf, steps, pgd):
  import flowpm_b200 as fpm
  from flowpm_b200 import tfpm
  cosmo = fpm.cosmology.Planck15()
  rng = np.random.default_rng(2)
  q = np.stack(np.indices((nc,) * 3), -1).reshape(-1, 3)
  s = rng.standard_normal((3, batch, nc**3, 3)) * 0.3
  s[0] += q
  s = torch.tensor(s.astype(np.float32), device='cuda')
  keep = s.clone()
  stages = np.linspace(0.2, 0.6, steps + 1)
  kw = dict(pm_nc_factor=bf)
  if pgd and steps:
    kw['pgdparams'] = [(0.01, 1.1, 7.0)] * steps
  a = fpm.nbody(cosmo, s, stages, nc, **kw)
  monkeypatch.setattr(tfpm, '_DIRECT_PARTICLES', 0)
  b = fpm.nbody(cosmo, s, stages, nc, **kw)
  assert torch.equal(s, keep)
  # the paint adds in any order: 2e-7 of the density a step, in a few steps
  for i in range(3):
    scale = max(1., float(a[i].abs().max()))
    assert float((a[i] - b[i]).abs().max()) < 2e-5 * scale
