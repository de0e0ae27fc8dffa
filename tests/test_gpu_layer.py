"""The native layer call behind the modules (`ocnn.nn.ConvLayer`): BatchNorm folded inside the kernels,
weights packed again when they change, copies and pickles of a module, the per-octree tables."""
import copy
import pickle

import pytest
import torch

import gpu_util as gu
from oracle import oracle as oc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ocnn():
  import ocnn as mod
  mod.set_key_bits(64)
  return mod


@pytest.fixture(scope='module')
def batch():
  _, merged, _ = gu.oracle_batch(gu.small_clouds(3, 3000, 500), 5, 2, 64)
  return gu.to_cuda_u8(merged), oc.OctreeView(merged)


def randomised(bn, seed):
  g = torch.Generator().manual_seed(seed)
  with torch.no_grad():
    for t, lo in ((bn.weight, 0.5), (bn.bias, -0.3), (bn.running_mean, -0.3), (bn.running_var, 0.5)):
      t.copy_(torch.rand(t.shape, generator=g) + lo)
  return bn


# (cin, cout, kernel, dtype): group mode, node mode, folded 1x1 (with a node count that leaves a tail on
# non-empty nodes), CUDA-core kernel
@pytest.mark.parametrize('cin,cout,ks,nempty', [
    (8, 16, [3], False), (64, 64, [3], False), (24, 40, [3], True), (32, 8, [1], False),
    (16, 32, [1], True), (64, 256, [1], False), (5, 7, [3], False)])
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16, torch.float16])
def test_batchnorm_in_the_epilogue(ocnn, batch, cin, cout, ks, nempty, dtype):
  octree, v = batch
  if dtype != torch.float32 and cin % 8:
    pytest.skip('16-bit layers take multiples of eight channels')
  d = 5
  h = int(v.nnum_nempty[d] if nempty else v.nnum[d])
  torch.manual_seed(cin + cout)
  x = torch.randn(1, cin, h, 1, device='cuda').to(dtype)
  res = torch.randn(1, cout, h, 1, device='cuda').to(dtype)
  if dtype != torch.float32:
    x = x.contiguous(memory_format=torch.channels_last)
    res = res.contiguous(memory_format=torch.channels_last)
  bn = randomised(torch.nn.BatchNorm2d(cout, 1e-3), 3).cuda().eval()
  if ks == [1]:
    layer = ocnn.OctreeConv1x1(cin, cout).cuda().eval()
    call = lambda *a: layer.run(x, *a)
  else:
    layer = ocnn.OctreeConv(d, cin, cout, ks, nempty=nempty).cuda().eval()
    call = lambda *a: layer._run(x, octree, *a)
  with torch.no_grad():
    for _ in range(2):                     # the second pass after the parameters have changed in place
      got = call(bn, res, True).float()
      want = torch.relu(bn(call().float()) + res.float())
      scale = float(want.abs().max())
      assert float((got - want).abs().max()) < (1e-5 if dtype == torch.float32 else 2e-2) * scale
      for p in list(layer.parameters()) + [bn.running_mean, bn.running_var]:
        p.mul_(1.25)


def test_copies_of_a_used_layer(ocnn, batch):
  octree, v = batch
  x = torch.randn(1, 8, int(v.nnum[5]), 1, device='cuda').to(torch.bfloat16)
  x = x.contiguous(memory_format=torch.channels_last)
  net = ocnn.OctreeConvBnRelu(5, 8, 16).cuda().eval()
  with torch.no_grad():
    want = net(x, octree)
    for other in (copy.deepcopy(net), pickle.loads(pickle.dumps(net))):
      assert torch.equal(other(x, octree), want)


def test_tables_follow_the_octree(ocnn, batch):
  """The inverse child table kept with an octree: per stream, and gone with the octree's content."""
  octree, v = batch
  other = torch.cuda.Stream()
  conv = ocnn.OctreeConv(5, 8, 8, nempty=True).cuda().eval()
  x = torch.randn(1, 8, int(v.nnum_nempty[5]), 1, device='cuda')
  with torch.no_grad():
    mine = octree.clone()
    want = conv(x, octree)
    assert torch.equal(conv(x, mine), want) and torch.equal(conv(x, mine), want)
    other.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(other):
      got = conv(x, mine)
    torch.cuda.current_stream().wait_stream(other)
    assert torch.equal(got, want)
    mine.copy_(octree)                     # the same storage, written to: the tables are made again
    assert torch.equal(conv(x, mine), want)


# (1x1 with cuDNN's and with our own weight gradient, sibling-group and node mode, deconvolution)
@pytest.mark.parametrize('kind,cin,cout,nempty', [
    ('conv1x1', 16, 32, False), ('conv1x1', 16, 64, False), ('conv', 8, 16, False), ('conv', 16, 8, True),
    ('deconv', 16, 8, False), ('deconv', 8, 8, True)])
@pytest.mark.parametrize('with_res', [False, True])
def test_training_block_is_the_modules_one_by_one(ocnn, batch, kind, cin, cout, nempty, with_res):
  octree, v = batch
  torch.manual_seed(cin + cout)
  h_in = h_out = int(v.nnum_nempty[4] if nempty else v.nnum[4])
  if kind == 'conv1x1':
    block = ocnn.OctreeConv1x1BnRelu(cin, cout, use_bias=with_res).cuda().train()
    args = ()
  elif kind == 'conv':
    block = ocnn.OctreeConvBnRelu(4, cin, cout, nempty=nempty).cuda().train()
    args = (octree,)
  else:
    block = ocnn.OctreeDeConvBnRelu(4, cin, cout, [3], 2, nempty).cuda().train()
    args = (octree,)
    h_out = int(v.nnum_nempty[5] if nempty else v.nnum[5])
  one = copy.deepcopy(block)
  one.bn.register_forward_hook(lambda *a: None)            # a hook inside: no single node
  data = torch.randn(1, cin, h_in, 1, device='cuda')
  res = torch.randn(1, cout, h_out, 1, device='cuda') if with_res else None
  g = torch.randn(1, cout, h_out, 1, device='cuda')
  got = []
  for b in (block, one):
    x = data.clone().requires_grad_()
    r = None if res is None else res.clone().requires_grad_()
    y = b(x, *args, residual=r)
    y.backward(g)
    got.append([y.detach(), x.grad] + ([] if r is None else [r.grad]) + [p.grad for p in b.parameters()] +
               [t.float() for t in b.bn.buffers()])
  assert len(got[0]) == len(got[1]) > 5
  for a, b in zip(*got):
    torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)
  with pytest.raises(ValueError):
    ocnn.OctreeConv1x1BnRelu(4, 4).cuda().train()(torch.ones(1, 4, 1, 1, device='cuda'))


@pytest.fixture(scope='module')
def sparse_level(ocnn):
  """About 97 k non-empty nodes at depth 7, a slab among scattered points: from 1 to 27 neighbours."""
  gen = torch.Generator().manual_seed(7)
  p = 0.99 * (2 * torch.rand(100000, 3, generator=gen) - 1)
  p[50000:] = p[50000:] * torch.tensor([1.0, 1.0, 0.02])
  n = torch.nn.functional.normalize(torch.randn(100000, 3, generator=gen), dim=1)
  octree = ocnn.octree_batch([ocnn.Points2Octree(7, 2)(ocnn.points_new(p, n, torch.zeros(0), torch.zeros(0)))]).cuda()
  return octree, int((ocnn.octree_property(octree, 'child', 7) >= 0).sum())


# (one and several 64-channel parts per tap, one and several taps per K-block, padded columns, slices of
# 256; 256 columns take the persistent kernel, fp32 the three-part one; the gradient its own gather)
@pytest.mark.parametrize('cin,cout', [(64, 64), (96, 96), (128, 104), (32, 72), (8, 64), (192, 512), (64, 256)])
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16])
def test_missing_neighbours_on_a_large_sparse_level(ocnn, sparse_level, cin, cout, dtype):
  octree, h = sparse_level
  torch.manual_seed(cin + cout)
  op = ocnn.OctreeConv(7, cin, cout, [3], 1, True).cuda().eval()
  x = torch.randn(1, cin, h, 1, device='cuda').to(dtype).contiguous(memory_format=torch.channels_last)
  res = torch.randn(1, cout, h, 1, device='cuda').to(dtype).contiguous(memory_format=torch.channels_last)
  bn = randomised(torch.nn.BatchNorm2d(cout, 1e-3), 3).cuda().eval()
  with torch.no_grad():
    op.weights.copy_(op.weights.to(dtype).float())
    z = op._run(x.float().contiguous(), octree)
    got, want = op._run(x, octree, bn, res, True).float(), torch.relu(bn(z) + res.float())
    assert float((got - want).abs().max() / want.abs().max()) < (1e-2 if dtype == torch.bfloat16 else 2e-3)


class _Tripled(torch.nn.Conv1d):
  def forward(self, x):
    return 3 * super().forward(x)


@pytest.mark.parametrize('cout', [24, 64])                 # torch's weight gradient, and our own
@pytest.mark.parametrize('block', [False, True])
def test_replaced_or_hooked_conv1d_is_called(ocnn, cout, block):
  """Training paths that pass the inner Conv1d by keep to the stock one."""
  layer = (ocnn.OctreeConv1x1BnRelu if block else ocnn.OctreeConv1x1)(16, cout).cuda().train()
  inner = layer.conv1x1 if block else layer
  x = torch.randn(1, 16, 500, 1, device='cuda', requires_grad=True)
  seen = []
  handle = inner.conv1x1.register_forward_pre_hook(lambda m, i: seen.append(m))
  layer(x)
  handle.remove()
  assert seen == [inner.conv1x1]
  tripled = _Tripled(16, cout, 1, bias=False).cuda()
  tripled.load_state_dict(inner.conv1x1.state_dict())
  y = inner(x)
  inner.conv1x1 = tripled
  torch.testing.assert_close(inner(x), 3 * y, rtol=1e-3, atol=1e-3)
  if block:
    want = torch.relu(layer.bn(inner(x)))
    torch.testing.assert_close(layer(x), want, rtol=1e-3, atol=1e-3)


def test_conv1d_of_another_width(ocnn):
  """The native side of a 1x1 layer follows a Conv1d of another shape."""
  layer = ocnn.OctreeConv1x1(16, 24).cuda().eval()
  with torch.no_grad():
    for cin, cout in [(16, 24), (16, 8), (32, 8)]:
      layer.conv1x1 = torch.nn.Conv1d(cin, cout, 1, bias=False).cuda()
      for dtype, tol in ((torch.float32, 1e-5), (torch.bfloat16, 1e-2)):
        x = torch.randn(1, cin, 300, 1, device='cuda').to(dtype).contiguous(memory_format=torch.channels_last)
        got = layer(x)
        ref = torch.einsum('oc,ch->oh', layer.conv1x1.weight[:, :, 0].double(), x.squeeze(0).squeeze(-1).double())
        assert got.shape == (1, cout, 300, 1)
        assert float((got.double().squeeze(0).squeeze(-1) - ref).norm() / ref.norm()) < tol


def test_another_parameter_at_the_same_place(ocnn, batch):
  """A parameter that is dropped for a new one of the same size, which the allocator puts where it lay."""
  octree, v = batch
  x = torch.randn(1, 64, int(v.nnum[4]), 1, device='cuda').to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
  layer = ocnn.OctreeConv(4, 64, 64).cuda().eval()
  layer.weights = torch.nn.Parameter(torch.randn(64, 64 * 27, device='cuda'))
  same = 0
  with torch.no_grad():
    for _ in range(8):
      before = layer.weights.data_ptr(), layer.weights._version
      layer(x, octree)
      del layer.weights
      layer.weights = torch.nn.Parameter(torch.randn(64, 64 * 27, device='cuda'))
      same += (layer.weights.data_ptr(), layer.weights._version) == before
      assert torch.equal(layer(x, octree), copy.deepcopy(layer)(x, octree))
  assert same > 0


def test_packed_weights_on_another_stream(ocnn, batch):
  """A second stream waits for the weights that the first one is still to pack."""
  octree, v = batch
  x = torch.randn(1, 64, int(v.nnum[4]), 1, device='cuda').to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
  layer = ocnn.OctreeConv(4, 64, 64).cuda().eval()
  ocnn.octree_property(octree, 'child', 4)                 # (the octree's header is read)
  side = torch.cuda.Stream()
  torch.cuda.synchronize()
  with torch.no_grad():
    torch.cuda._sleep(20_000_000)                          # about 10 ms on the first stream
    mine = layer(x, octree)
    with torch.cuda.stream(side):
      theirs = layer(x, octree)
    torch.cuda.synchronize()
    assert torch.equal(mine, theirs)
    # packed inside a capture: the graph's own, not kept for later calls
    fresh = copy.deepcopy(layer)
    fresh.weights.mul_(2.0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
      y = fresh(x, octree)
    eager = fresh(x, octree)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, eager)
    # captured with weights that were packed before, on this stream or another: the graph's image stays
    for warm_up in (torch.cuda.current_stream(), side):
      with torch.cuda.stream(warm_up):
        eager = fresh(x, octree)
      torch.cuda.synchronize()
      later = torch.cuda.CUDAGraph()
      with torch.cuda.graph(later, stream=side):
        z = fresh(x, octree)
      fresh.weights.mul_(2.0)
      double = fresh(x, octree)
      for _ in range(4):
        torch.randn_like(layer.weights)    # (would take the place of an image that is given back)
      later.replay()
      torch.cuda.synchronize()
      assert torch.equal(z, eager) and not torch.equal(double, eager)
      fresh.weights.mul_(0.25)


def test_parameter_read_as_another_view(ocnn, batch):
  """The same storage, transposed, is another set of weights."""
  octree, v = batch
  x = torch.randn(1, 64, int(v.nnum[4]), 1, device='cuda').to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
  layer = ocnn.OctreeConv1x1(64, 64).cuda().eval()
  weight = layer.conv1x1.weight.detach()
  with torch.no_grad():
    layer(x)
    layer.conv1x1.weight.data = weight.transpose(0, 1)
    assert torch.equal(layer(x), copy.deepcopy(layer)(x))
