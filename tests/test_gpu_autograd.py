"""What looks at a 1x1 training layer or block besides one backward pass: second derivatives, forward mode,
functorch transforms, tracing, saved-tensor hooks, against the same torch modules (Conv1d, BatchNorm2d, ReLU)."""
import copy

import pytest
import torch
import torch.autograd.forward_ad as fw

import gpu_util as gu
from oracle import oracle as oc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ocnn():
  import ocnn as mod
  mod.set_key_bits(64)
  return mod


@pytest.fixture(autouse=True)
def no_tf32():
  old = torch.backends.cudnn.allow_tf32
  torch.backends.cudnn.allow_tf32 = False
  yield
  torch.backends.cudnn.allow_tf32 = old


def plain(block, x, residual=None):
  """The block's values through torch's modules."""
  conv = block.conv1x1
  conv = getattr(conv, 'conv1x1', conv)
  y = conv(x.squeeze(-1)).unsqueeze(-1)
  if hasattr(block, 'bn'):
    y = block.bn(y)
    y = y if residual is None else y + residual
    y = torch.relu(y) if block.with_relu else y
  return y


def close(a, b, tol=2e-4, scale=0.0):
  """scale: the size of the terms of a sum that is 0 but for their rounding (a bias ahead of a BatchNorm)."""
  a, b = a.detach(), b.detach()
  assert float((a - b).norm()) <= tol * float(b.norm()) + 1e-6 * (1 + scale)


def make(ocnn, kind, cout, bias=False):
  torch.manual_seed(cout)
  cls = {'layer': ocnn.OctreeConv1x1, 'bn': ocnn.OctreeConv1x1Bn, 'bnrelu': ocnn.OctreeConv1x1BnRelu}[kind]
  return cls(16, cout, bias).cuda().train()


@pytest.mark.parametrize('kind', ['layer', 'bn', 'bnrelu'])
@pytest.mark.parametrize('cout,bias', [(24, False), (64, True)])       # torch's weight gradient, and our own
def test_second_derivatives(ocnn, kind, cout, bias):
  block = make(ocnn, kind, cout, bias)
  results = []
  for fn in (lambda x, r: block(x, residual=r) if kind != 'layer' else block(x), lambda x, r: plain(block, x, r)):
    torch.manual_seed(1)
    x = torch.randn(1, 16, 200, 1, device='cuda', requires_grad=True)
    res = torch.randn(1, cout, 200, 1, device='cuda', requires_grad=True)
    g = torch.randn(1, cout, 200, 1, device='cuda', requires_grad=True)
    leaves = [x] + list(block.parameters()) + ([res] if kind != 'layer' else [])
    first = torch.autograd.grad(fn(x, res), leaves, g, create_graph=True)
    penalty = sum((t * torch.linspace(0.5, 1.5, t.numel(), device='cuda').view_as(t)).pow(2).sum() for t in first)
    second = torch.autograd.grad(penalty, leaves + [g], allow_unused=True)
    results.append((first, second))
  for order, tol in ((0, 2e-4), (1, 2e-3)):
    scale = max(float(t.detach().norm()) for t in results[1][order] if t is not None)
    for got, want in zip(results[0][order], results[1][order]):
      zero = torch.zeros((), device='cuda')
      close(zero if got is None else got, zero if want is None else want, tol, scale)


@pytest.mark.parametrize('kind', ['layer', 'bnrelu'])
@pytest.mark.parametrize('cout', [24, 64])
def test_forward_mode_transforms_and_tracing(ocnn, kind, cout):
  block = make(ocnn, kind, cout)
  x, t = torch.randn(2, 1, 16, 200, 1, device='cuda')
  ref = copy.deepcopy(block)
  for p in block.parameters():
    p.requires_grad_(True)
  with fw.dual_level():
    got = fw.unpack_dual(block(fw.make_dual(x, t)))
    want = fw.unpack_dual(plain(ref, fw.make_dual(x, t)))
  close(got.primal, want.primal)
  close(got.tangent, want.tangent)
  if kind == 'layer':                      # (a BatchNorm's running statistics cannot be updated in a transform)
    params = dict(block.named_parameters())
    grads = torch.func.grad(lambda p: torch.func.functional_call(block, p, (x,)).pow(2).sum())(params)
    y = plain(ref, x).pow(2).sum()
    for got, want in zip(grads.values(), torch.autograd.grad(y, list(ref.parameters()))):
      close(got, want, 2e-3)
  traced = torch.jit.trace(block, (x,), check_trace=False)
  close(traced(x), block(x))


def test_saved_tensor_hooks_see_a_block(ocnn):
  block = make(ocnn, 'bnrelu', 24)
  x = torch.randn(1, 16, 200, 1, device='cuda', requires_grad=True)
  want = torch.autograd.grad(block(x).sum(), [x] + list(block.parameters()))
  with torch.autograd.graph.save_on_cpu():
    y = block(x)
  got = torch.autograd.grad(y.sum(), [x] + list(block.parameters()))
  for a, b in zip(got, want):
    assert torch.equal(a, b)


@pytest.mark.parametrize('deconv', [False, True])
def test_first_derivatives_of_an_octree_block_under_create_graph(ocnn, deconv):
  """A convolution block's gradients are the same with and without a graph of them."""
  _, merged, _ = gu.oracle_batch(gu.small_clouds(2, 2000, 500), 4, 2, 64)
  octree, v = gu.to_cuda_u8(merged), oc.OctreeView(merged)
  block = (ocnn.OctreeDeConvBnRelu if deconv else ocnn.OctreeConvBnRelu)(4, 8, 24).cuda().train()
  h = int(v.nnum[4])
  x = torch.randn(1, 8, h, 1, device='cuda', requires_grad=True)
  res = torch.randn(1, 24, h, 1, device='cuda', requires_grad=True)
  g = torch.randn(1, 24, h, 1, device='cuda', requires_grad=True)
  leaves = [x, res] + list(block.parameters())
  want = torch.autograd.grad(block(x, octree, residual=res), leaves, g)
  got = torch.autograd.grad(block(x, octree, residual=res), leaves, g, create_graph=True)
  for a, b in zip(got, want):
    close(a.detach(), b, 1e-5)
  # through the BatchNorm's parameters the second derivatives are torch's
  one = copy.deepcopy(block)
  one.bn.register_forward_hook(lambda *a: None)
  second = []
  for b in (block, one):
    gw, = torch.autograd.grad(b(x, octree, residual=res), b.bn.weight, g, create_graph=True)
    second.append(torch.autograd.grad(gw.pow(2).sum(), g)[0])
  close(second[0], second[1])


def test_a_block_is_called_without_a_count_of_batches(ocnn):
  """The native block's count is an optional last argument: left out, the rest is as with it."""
  block = make(ocnn, 'bnrelu', 24)
  conv, bn = block.conv1x1.conv1x1, block.bn
  x = torch.randn(1, 16, 200, 1, device='cuda')
  args = lambda: (x, conv.weight, conv.bias, bn.weight, bn.bias, None, torch.zeros(24, device='cuda'),
                  torch.ones(24, device='cuda'), 0.01, 1e-3, None, 2, 0, 24, [1], 1, False, True)
  seen = torch.zeros((), dtype=torch.int64, device='cuda')
  assert torch.equal(ocnn.nn.train_block(*args()), ocnn.nn.train_block(*args(), seen)) and int(seen) == 1


@pytest.mark.parametrize('count', ['gpu', 'cpu', 'int32', 'two'])
@pytest.mark.parametrize('residual', ['none', 'rows', 'transposed'])       # (the last: added by torch's operator)
def test_a_block_counts_batches_as_a_write(ocnn, count, residual):
  """num_batches_tracked goes up by one and so does its version, wherever and however it is held."""
  block = make(ocnn, 'bnrelu', 24)
  seen = {'gpu': lambda: torch.tensor(5, device='cuda'), 'cpu': lambda: torch.tensor(5),
          'int32': lambda: torch.tensor(5, dtype=torch.int32, device='cuda'),
          'two': lambda: torch.tensor([5, 9], device='cuda')}[count]()
  block.bn.num_batches_tracked = seen
  x = torch.randn(1, 16, 200, 1, device='cuda')
  res = {'none': None, 'rows': torch.randn(1, 24, 200, 1, device='cuda'),
         'transposed': torch.randn(1, 200, 24, 1, device='cuda').transpose(1, 2)}[residual]
  want, version = seen + 1, seen._version
  block(x, residual=res)
  assert torch.equal(seen, want) and seen._version == version + 1
