"""`ocnn.ResNet` with another classification header than its own: whatever stands there is what runs, and
the one-launch form of pool + Linear keeps out of its way."""
import copy

import pytest
import torch
from torch import nn

import gpu_util as gu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def setup():
  import ocnn
  ocnn.set_key_bits(64)
  _, merged, _ = gu.oracle_batch(gu.small_clouds(3, 2000, 300), 4, 2, 64)
  octree = gu.to_cuda_u8(merged)
  torch.manual_seed(0)
  net = ocnn.ResNet(4, 8, 10, 1).cuda().eval()
  data = ocnn.nn.feature_node_major(octree, 8, True)
  stock = net.header
  net.header = nn.Identity()
  with torch.no_grad():
    feature = net(octree, data)
  assert feature.dtype == torch.float32 and feature.shape[1] == 256
  yield ocnn, net, octree, data, stock, feature
  net.header = stock


class Doubled(nn.Linear):
  def forward(self, x):
    return 2 * super().forward(x)


def headers(ocnn, stock):
  pool, fc = stock
  pool3 = ocnn.FullOctreeGlobalPool(depth=2)
  pool3.octree2voxel = nn.Sequential(ocnn.FullOctree2Voxel(2), nn.ReLU())
  return {'stock': stock, 'single': pool, 'one element': nn.Sequential(pool), 'no weight': nn.Sequential(pool, nn.ReLU()),
          'longer': nn.Sequential(pool, fc, nn.LogSoftmax(dim=1)), 'subclass': nn.Sequential(pool, Doubled(256, 7).cuda()),
          'other pool': nn.Sequential(pool3, fc), 'deeper pool': nn.Sequential(ocnn.FullOctreeGlobalPool(depth=1), fc),
          'no bias': nn.Sequential(pool, nn.Linear(256, 5, bias=False).cuda())}


@pytest.mark.parametrize('name', ['stock', 'single', 'one element', 'no weight', 'longer', 'subclass', 'other pool',
                                  'deeper pool', 'no bias'])
def test_header_that_stands_there_runs(setup, name):
  ocnn, net, octree, data, stock, feature = setup
  net.header = headers(ocnn, stock)[name]
  with torch.no_grad():
    got, want = net(octree, data), net.header(feature)
    torch.testing.assert_close(got, want, rtol=1e-3, atol=1e-3 * float(want.abs().max()))
    exact = net.header(net_features(net, octree))
    torch.testing.assert_close(net(octree, octree_data(ocnn, octree)), exact)


def octree_data(ocnn, octree):
  data = ocnn.octree_property(octree, 'feature', 4)
  return torch.cat([data, data.new_zeros(1, 5, data.shape[2], 1)], 1)


def net_features(net, octree):
  """The fp32 network's features, whatever its header."""
  import ocnn
  header, net.header = net.header, nn.Identity()
  out = net(octree, octree_data(ocnn, octree))
  net.header = header
  return out


def test_training_runs_a_replaced_header(setup):
  ocnn, net, octree, data, stock, feature = setup
  net.header = nn.Identity()
  out = copy.deepcopy(net).train()(octree, octree_data(ocnn, octree))     # (a copy: it updates its statistics)
  assert out.shape == feature.shape


def test_hooks_and_gradients_of_the_header(setup):
  ocnn, net, octree, data, stock, feature = setup
  net.header = stock
  with torch.no_grad():
    plain = net(octree, data)
    seen = []
    for module in (stock, stock[0], stock[0].octree2voxel, stock[1]):
      handle = module.register_forward_hook(lambda m, i, o: seen.append(m))
      net(octree, data)
      handle.remove()
      assert seen and seen[-1] is module
    handle = nn.modules.module.register_module_forward_hook(lambda m, i, o: seen.append(m))
    net(octree, data)
    handle.remove()
    assert any(m is stock[1] for m in seen[4:])
  net.requires_grad_(False)
  stock[1].requires_grad_(True)            # a frozen network, its Linear being trained
  logits = net(octree, data)
  torch.testing.assert_close(logits.detach(), plain, rtol=1e-3, atol=1e-3)
  grad, = torch.autograd.grad(logits.sum(), stock[1].weight)
  pooled = feature.view(256, -1, 64).mean(2).sum(1)
  torch.testing.assert_close(grad[0], pooled, rtol=1e-3, atol=1e-3)
  net.requires_grad_(True)
