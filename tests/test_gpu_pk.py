"""Power-spectrum binning at the sizes where its branches change: odd and
self-conjugate axes, modes on the bin edges, and bin counts on both sides of
the histograms' shared-memory limits."""
import numpy as np
import pytest
import torch

from oracle import pm as opm

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def fpm():
  import flowpm_b200
  return flowpm_b200


# box = 2 pi: |k| of the axis modes is a whole number, on the edges of
# kmin = dk = 1; dk chosen for 511 / 512 (histogram per warp / per block) and
# 4095 / 4096 edges (per block / none) on a mesh of 16
@pytest.mark.parametrize('shape,batch,kmin,dk', [
    ((16, 16, 16), 2, 1.0, 1.0), ((9, 8, 7), 1, 1.0, 1.0),
    ((5, 33, 64), 2, 1.0, 0.5), ((2, 3, 66), 1, 0.5, 0.25),
    ((64, 2, 31), 1, 0.3, 0.37), ((1, 16, 16), 1, 0.0, 0.5),
    ((16, 16, 16), 1, 1.0, 7.0 / 510.5), ((16, 16, 16), 1, 1.0, 7.0 / 511.5),
    ((16, 16, 16), 1, 1.0, 7.0 / 4094.5),
    ((16, 16, 16), 2, 1.0, 7.0 / 4095.5)])
def test_power_spectrum_edges(fpm, shape, batch, kmin, dk):
  rng = np.random.default_rng(7)
  f = rng.standard_normal((batch,) + shape).astype(np.float32)
  box = np.array([2 * np.pi] * 3)
  if len(fpm.pk.pk_edges(list(shape), box, kmin, dk)) < 2:
    pytest.skip('fewer than two edges')
  kb, p = fpm.power_spectrum(f, kmin=kmin, dk=dk, boxsize=box)
  with np.errstate(invalid='ignore'):
    kr, r = opm.power_spectrum(torch.tensor(f, dtype=torch.float64),
                               kmin=kmin, dk=dk, boxsize=box)
  np.testing.assert_array_equal(kb, kr)
  p, r = p.cpu().numpy(), r.numpy()
  assert p.shape == r.shape
  # empty bins are 0 / 0 on both sides, so the bins hold the same modes
  np.testing.assert_array_equal(np.isnan(p), np.isnan(r))
  # a mode F carries the transform's error, about 4e-7 of the rms mode, and
  # |F|^2 twice that times |F|
  scale = np.nanmax(r)
  np.testing.assert_allclose(p, r, rtol=1e-5, atol=4e-6 * scale)
