"""One cached plan used from two streams: calls that no longer wait for their
stream stay in order on the plan's tables and scratch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nc', [16, 20])
def test_plan_on_two_streams(cuda, nc):
  import flowpm_b200 as fpm
  cosmo = fpm.cosmology.Planck15()
  rng = np.random.default_rng(11)
  lin = [torch.tensor(rng.standard_normal((1, nc, nc, nc)).astype(np.float32),
                      device='cuda') for _ in range(2)]
  r = torch.tensor(rng.standard_normal((3, 1, nc**3, 3)).astype(np.float32),
                   device='cuda')

  def run(k, grad):
    x = lin[k].detach().clone().requires_grad_(grad)
    st = fpm.lpt_init(cosmo, x, 0.1 + 0.1 * k, 2)
    if not grad:
      return st
    st = fpm.nbody(cosmo, st, [0.2, 0.3 + 0.1 * k, 0.6], nc)
    return torch.autograd.grad((st * r).sum(), x)[0]

  for grad in (False, True):
    want = [run(k, grad) for k in range(2)]
    torch.cuda.synchronize()
    got = []
    for k in range(2):
      with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda._sleep(20000000)  # what follows queues up behind 10 ms
        got.append(run(k, grad))
    torch.cuda.synchronize()
    for g, w in zip(got, want):
      # the paint adds in any order: 1e-6 of the density in each of a few
      # steps, and as much of a gradient
      g, w = g.cpu().numpy(), w.cpu().numpy()
      np.testing.assert_allclose(g, w, rtol=0, atol=1e-4 * np.abs(w).max())
