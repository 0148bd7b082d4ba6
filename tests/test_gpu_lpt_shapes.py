"""The fused 2LPT passes against the library-transform path and in 64 bits, at
every axis length they are instantiated for, for several simulations and both
orders; unaligned arrays take the general path."""
import numpy as np
import pytest
import torch

from oracle import pm as opm

pytestmark = pytest.mark.gpu

COEF = [0.7, -0.2, 0.31, 0.17, 0.45, -0.6]


def _lpt(dims, lin, order, flags, name, offset=0):
  from flowpm_b200 import _lib
  from flowpm_b200._plans import Plan
  plan = Plan(dims, flags=flags | _lib.FPM_PLAN_LPT)
  n = lin.numel()
  buf = torch.empty(n + 4, device='cuda')
  x = buf[offset:offset + n].copy_(lin.reshape(-1))
  out = torch.empty((3, n, 3), device='cuda')
  try:
    _lib.call(name, plan.handle, _lib.ptr(x),
              _lib.dvec(COEF * len(dims)), order, _lib.ptr(out[0]),
              _lib.ptr(out[1]), _lib.ptr(out[2]), _lib.stream_ptr())
    torch.cuda.synchronize()
    return out
  finally:
    plan.close()


@pytest.mark.parametrize('shape', [
    (16, 16, 16), (32, 16, 64), (64, 128, 32), (128, 64, 16), (16, 32, 128),
    (16, 256, 256), (256, 16, 64), (32, 64, 512), (16, 512, 32),
    (512, 32, 16)])
@pytest.mark.parametrize('count,order', [(1, 2), (3, 2), (2, 1)])
def test_fused_lpt(cuda, shape, count, order):
  from flowpm_b200 import _lib
  dims = [tuple(shape) + (1,)] * count
  n = int(np.prod(shape))
  g = torch.Generator(device='cuda').manual_seed(5)
  lin = torch.randn((count, n), generator=g, device='cuda')
  a = _lpt(dims, lin, order, 0, 'fpm_lpt_init')
  b = _lpt(dims, lin, order, _lib.FPM_PLAN_CUFFT, 'fpm_lpt_init')
  c = _lpt(dims, lin, order, 0, 'fpm_lpt_init', offset=1)
  # transforms of up to 2^22 values, about log2(n) roundings of 6e-8 of the
  # rms each; a second-order displacement carries its source's as well
  scale = b.abs().amax(dim=(1, 2))
  assert bool(((a - b).abs().amax(dim=(1, 2)) < 2e-5 * scale).all())
  assert bool(((c - b).abs().amax(dim=(1, 2)) < 2e-5 * scale).all())
  s = _lpt(dims, lin, order, 0, 'fpm_lpt_state')
  q = torch.tensor(np.stack(np.indices(shape), -1).reshape(1, -1, 3),
                   dtype=torch.float32, device='cuda')
  assert torch.equal(s[1:], a[1:])
  assert torch.equal(s[0].reshape(count, -1, 3), a[0].reshape(
      count, -1, 3) + q)


@pytest.mark.parametrize('shape', [(32, 16, 64), (64, 64, 64)])
def test_fused_lpt_64_bits(cuda, shape):
  """No further from 64 bits than twice the library-transform path."""
  from flowpm_b200 import _lib
  dims = [tuple(shape) + (1,)]
  lin = torch.randn((1,) + shape, device='cuda',
                    generator=torch.Generator(device='cuda').manual_seed(6))
  a = _lpt(dims, lin, 2, 0, 'fpm_lpt_init').double().cpu()
  b = _lpt(dims, lin, 2, _lib.FPM_PLAN_CUFFT, 'fpm_lpt_init').double().cpu()
  x = np.fft.rfftn(lin[0].double().cpu().numpy())
  k = opm.fftk(shape)
  lap = opm.laplace_kernel(k)
  g = [opm.gradient_kernel(k, d) for d in range(3)]
  inv = lambda f: np.fft.irfftn(f, s=shape)
  psi = [inv(x * lap * g[d]) for d in range(3)]
  p = [inv(x * lap * g[d] * g[d]) for d in range(3)]
  q = [inv(x * lap * g[i] * g[j]) for i, j in ((1, 2), (2, 0), (0, 1))]
  src = 3. / 7. * (p[1] * p[2] + p[2] * p[0] + p[0] * p[1] -
                   q[0]**2 - q[1]**2 - q[2]**2)
  y = np.fft.rfftn(src)
  psi2 = [inv(y * lap * g[d]) for d in range(3)]
  p1 = np.stack(psi, -1).reshape(-1, 3)
  p2 = np.stack(psi2, -1).reshape(-1, 3)
  c = np.array(COEF, np.float32).astype(np.float64)
  for i, (u, v) in enumerate(((1., 1.), (c[2], c[3]), (c[4], c[5]))):
    r = torch.tensor(u * c[0] * p1 + v * c[1] * p2)
    ea, eb = (a[i] - r).norm() / r.norm(), (b[i] - r).norm() / r.norm()
    assert ea < 2 * eb + 1e-7, (float(ea), float(eb))
