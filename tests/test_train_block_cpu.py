"""The native block node (`ocnn.nn.train_block`) on a 1x1 layer whose tensors lie in host memory: torch's operators."""
import pytest
import torch

import ocnn

EPS32 = 2.0 ** -24


@pytest.mark.parametrize('cout', [24, 96])               # (96: on the GPU with this library's weight gradient)
@pytest.mark.parametrize('relu', [False, True])
@pytest.mark.parametrize('with_res', [False, True])
@pytest.mark.parametrize('needs_data', [False, True])
def test_a_1x1_block_in_host_memory(cout, relu, with_res, needs_data):
  torch.manual_seed(cout)
  conv, bn = torch.nn.Conv1d(16, cout, 1), torch.nn.BatchNorm2d(cout, 1e-3, 0.01)
  x = torch.randn(1, 16, 50, 1, requires_grad=needs_data)
  res = torch.randn(1, cout, 50, 1, requires_grad=True) if with_res else None
  g = torch.randn(1, cout, 50, 1)
  wrt = [t for t in (x, res, conv.weight, bn.weight, bn.bias) if t is not None and t.requires_grad]
  y = bn(conv(x.squeeze(-1)).unsqueeze(-1))
  y = y + res if with_res else y
  want = torch.relu(y) if relu else y
  grads = torch.autograd.grad(want, wrt, g)
  mean, var, seen = torch.zeros(cout), torch.ones(cout), torch.zeros((), dtype=torch.int64)
  got = ocnn.nn.train_block(x, conv.weight, conv.bias, bn.weight, bn.bias, res, mean, var, 0.01, 1e-3, None, 2, 0, cout,
                            [1], 1, False, relu, seen)
  # the same operators; torch may choose another order for the 17 terms of a product and the 50 rows of a sum
  assert torch.allclose(got, want, rtol=16 * EPS32, atol=16 * EPS32)
  assert torch.equal(mean, bn.running_mean) and torch.equal(var, bn.running_var) and int(seen) == 1
  for a, b in zip(torch.autograd.grad(got, wrt, g), grads):
    assert torch.allclose(a, b, rtol=0, atol=64 * EPS32 * float(b.abs().max()))
