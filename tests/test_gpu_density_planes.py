"""Density planes where the row pairs, the modulus and the batch change form:
odd and tiny planes, positions up to three periods outside the box, several
batch entries, overlapping slabs and more slabs than one library call takes.
Positions are dyadic and the rotation a permutation, so that both sides find
the same cells and exact weights."""
import numpy as np
import pytest
import torch

from oracle import planes as opl

pytestmark = pytest.mark.gpu

PERM = np.array([[0, 0, 1], [1, 0, 0], [0, 1, 0]], np.float32)


@pytest.mark.parametrize('res', [1, 2, 3, 5, 8, 37])
@pytest.mark.parametrize('batch,npart', [(1, 1), (3, 700)])
@pytest.mark.parametrize('rot', [False, True])
@pytest.mark.parametrize('nplanes', [3, 66])
def test_density_planes(cuda, res, batch, npart, rot, nplanes):
  import flowpm_b200 as fpm
  nc, rng = 16, np.random.default_rng(res)
  st = rng.integers(-45 * 16, 48 * 16, (2, batch, npart, 3)) / 16.
  st[0, :, ::3] = np.mod(st[0, :, ::3], nc)
  st = st.astype(np.float32)
  centers = np.linspace(1., 15., nplanes)
  width = 6.0  # overlapping slabs
  g = rng.integers(-8, 9, (batch, nplanes, res, res)).astype(np.float32)
  kw = dict(rotation=PERM if rot else None,
            shift=np.array([0.25, 0.5, 0.125], np.float32) if rot else None)
  s = torch.tensor(st, device='cuda', requires_grad=True)
  out = fpm.raytracing.density_planes(s, nc, centers, width, res, **kw)
  (gs,) = torch.autograd.grad(out, s, torch.tensor(g, device='cuda'))
  so = torch.tensor(st, dtype=torch.float64, requires_grad=True)
  ref = torch.stack([opl.density_plane(so, nc, c, width, res, **kw)
                     for c in centers], dim=1)
  (gr,) = torch.autograd.grad(ref, so, torch.tensor(g, dtype=torch.float64))
  # exact sums; a division each (6e-8), and one more in the gradient's
  # scale, summed over the slabs of a particle
  np.testing.assert_allclose(out.detach().cpu().numpy(), ref.detach().numpy(),
                             rtol=1e-6, atol=1e-6 * float(ref.abs().max()))
  np.testing.assert_allclose(gs.cpu().numpy(), gr.numpy(), rtol=1e-6,
                             atol=1e-5 * max(1e-3, float(gr.abs().max())))
