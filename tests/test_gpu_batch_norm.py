"""The kernels around a training block's BatchNorm (`ocnn_batch_norm_backward`, `ocnn_batch_norm_finish`) against
torch's in 64 bits: slices with and without a remainder, clusters of one to eight CTAs, slices beyond shared
memory, data off a 16-byte boundary."""
import ctypes

import pytest
import torch

import ocnn

pytestmark = pytest.mark.gpu
EPS32 = 2.0 ** -24


def call(name, *args):
  lib = ctypes.CDLL(ocnn.LIBRARY)
  conv = lambda a: ctypes.c_void_p(a.data_ptr()) if isinstance(a, torch.Tensor) else \
      (ctypes.c_void_p(None) if a is None else a if isinstance(a, ctypes.c_int64) else ctypes.c_int(a))
  stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
  assert getattr(lib, name)(*[conv(a) for a in args], stream) == 0


def placed(t, shift):
  """The same values `shift` floats behind a 16-byte boundary."""
  return torch.empty(t.numel() + shift, device='cuda')[shift:].view(t.shape).copy_(t)


@pytest.mark.parametrize('channels,rows,shift', [
    (1, 2, 0), (3, 5, 0), (7, 1024, 1), (64, 4095, 0), (5, 4096, 0), (33, 16388, 2), (2, 40001, 0), (300, 8200, 0),
    (2, 500000, 0)])                       # the last: more than eight CTAs' shared memory holds
@pytest.mark.parametrize('relu', [False, True])
def test_gradient_against_64_bits(channels, rows, shift, relu):
  gen = torch.Generator('cuda').manual_seed(rows + channels)
  rand = lambda *s: torch.randn(*s, device='cuda', generator=gen)
  x = placed(rand(channels, rows) + 30 * rand(channels, 1), shift)
  gy, w = placed(rand(channels, rows), shift), rand(channels)
  x64 = x.double()
  mean, invstd = x64.mean(1).float(), (1 / (x64.var(1, unbiased=False) + 1e-3).sqrt()).float()
  out = placed(rand(channels, rows), shift) if relu else None
  g64 = torch.where(out > 0, gy, torch.zeros_like(gy)).double() if relu else gy.double()
  xhat = (x64 - mean.double()[:, None]) * invstd.double()[:, None]
  want = (g64 - g64.mean(1, keepdim=True) - xhat * (g64 * xhat).mean(1, keepdim=True)) * \
      (w.double() * invstd.double())[:, None]
  gx, gw, gb = placed(torch.empty_like(x), shift), torch.empty_like(w), torch.empty_like(w)
  call('ocnn_batch_norm_backward', x, gy, out, gx, channels, rows, w, mean, invstd, gw, gb)
  # five operations, each rounded once, on terms no larger than |g| + |mean| + |xhat * mean(g xhat)|
  terms = g64.abs() + g64.mean(1, keepdim=True).abs() + (xhat * (g64 * xhat).mean(1, keepdim=True)).abs()
  assert bool(((gx.double() - want).abs() <= 8 * EPS32 * terms * (w.double() * invstd.double()).abs()[:, None]).all())
  # one rounding of a sum in 64 bits
  assert bool(((gb.double() - g64.sum(1)).abs() <= 2 * EPS32 * g64.sum(1).abs() + 1e-12 * rows).all())
  dot = (g64 * xhat).sum(1)
  assert bool(((gw.double() - dot).abs() <= 2 * EPS32 * dot.abs() + 1e-10 * rows).all())


@pytest.mark.parametrize('count,shift', [(0, 0), (1, 0), (4, 1), (1023, 0), (4096, 0), (300001, 2)])
@pytest.mark.parametrize('relu', [False, True])
@pytest.mark.parametrize('with_res', [False, True])
def test_finish_is_torchs_addition_and_relu(count, shift, relu, with_res):
  y = placed(torch.randn(count, device='cuda'), shift)
  if count > 4:
    y[2], y[3], y[4] = float('nan'), float('inf'), -float('inf')
  res = placed(torch.randn(count, device='cuda'), shift) if with_res else None
  want = y if res is None else y + res
  want = torch.relu(want) if relu else want.clone()
  seen = torch.full((), 2 ** 40, dtype=torch.int64, device='cuda')
  call('ocnn_batch_norm_finish', y, res, ctypes.c_int64(count), int(relu), seen)
  torch.testing.assert_close(y, want, rtol=0, atol=0, equal_nan=True)
  assert int(seen) == 2 ** 40 + 1
