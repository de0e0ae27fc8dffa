"""fp32 layers on the tensor cores (three bf16 parts per value) and on whole sibling groups: every width of
the accumulator tile, more than one slice of output channels, K splits, chunk remainders, node counts
that do not fill a tile, against the column formulation in float64."""
import ctypes

import numpy as np
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
def octree(ocnn):
  _, merged, _ = gu.oracle_batch(gu.small_clouds(3, 3000, 500), 5, 2, 64)
  return gu.to_cuda_u8(merged), oc.OctreeView(merged)


@pytest.fixture(scope='module')
def big_octree(ocnn):
  """A level large enough for two groups per warp and several tiles per CTA."""
  _, merged, _ = gu.oracle_batch(gu.small_clouds(12, 6000, 500), 6, 2, 64)
  return gu.to_cuda_u8(merged), oc.OctreeView(merged)


def columns(ocnn, x, octree, d, nempty):
  return ocnn.nn.octree2col(x, octree, d, [3, 3, 3], 1, nempty).flatten(0, 1).double()


def off(got, want):
  return float((got.double() - want).norm() / want.norm())


# (cin, cout): each NG = cout / 16 of conv_f32_kernel, a slice boundary, channel counts that leave a
# K-block or an 8-channel chunk unfilled; few channels stay on the group kernel
CHANNELS = [(3, 5), (3, 64), (16, 16), (33, 16), (40, 32), (24, 48), (64, 64), (72, 80), (9, 96), (32, 112),
            (64, 128), (40, 130), (17, 257)]


@pytest.mark.parametrize('cin,cout', CHANNELS)
@pytest.mark.parametrize('depth,nempty,node_major', [(5, False, False), (5, True, False), (5, True, True), (2, False, True)])
def test_forward(ocnn, octree, cin, cout, depth, nempty, node_major):
  tree, v = octree
  h = int(v.nnum_nempty[depth] if nempty else v.nnum[depth])
  torch.manual_seed(cin * cout)
  x, w = torch.randn(1, cin, h, 1, device='cuda'), torch.randn(cout, cin * 27, device='cuda') * 0.1
  want = (w.double() @ columns(ocnn, x, tree, depth, nempty)).view(1, cout, h, 1)
  xin = x.contiguous(memory_format=torch.channels_last) if node_major else x
  got = ocnn.octree_conv(xin, w, tree, depth, cout, [3, 3, 3], 1, nempty)
  assert off(got, want) < 6e-7 and gu.rel_err(gu.to_np(got), want.view(cout, h).cpu().numpy()) < 1e-5
  chain = ocnn.nn.octree_conv(xin, w, tree, depth, cout, [3, 3, 3], 1, nempty, True)
  assert off(chain, want) < 2e-6


@pytest.mark.parametrize('cin,cout', [(3, 16), (4, 64), (20, 12), (32, 40), (64, 96)])
def test_forward_and_gradients_of_a_big_level(ocnn, big_octree, cin, cout):
  tree, v = big_octree
  d, h = 6, int(v.nnum[6])
  assert h > 2 * 148 * 16 * 8
  torch.manual_seed(cin)
  x, w = torch.randn(1, cin, h, 1, device='cuda'), torch.randn(cout, cin * 27, device='cuda') * 0.1
  g = torch.randn(1, cout, h, 1, device='cuda')
  col = columns(ocnn, x, tree, d, False)
  want = (w.double() @ col).view(1, cout, h, 1)
  for chain in (False, True):
    assert off(ocnn.nn.octree_conv(x, w, tree, d, cout, [3, 3, 3], 1, False, chain), want) < 2e-6
  gx, gw = ocnn.nn.octree_conv_grad(x, w, tree, g, d, cout, [3, 3, 3], 1, False)
  assert off(gw, g.view(cout, h).double() @ col.t()) < 2e-6
  gcol = (w.double().t() @ g.view(cout, h).double()).view(cin, 27, h).float()
  want = ocnn.nn.col2octree(gcol, tree, d, [3, 3, 3], 1, False).double()
  assert off(gx, want) < 2e-6
  only = ocnn.nn.octree_conv_grad(x, w, tree, g, d, cout, [3, 3, 3], 1, False, False, True)
  assert only[0] is None and torch.equal(only[1], gw)


@pytest.mark.parametrize('cin,cout', [(3, 5), (8, 32), (40, 33), (16, 64), (64, 96), (24, 128), (130, 257)])
@pytest.mark.parametrize('rows', [1, 31, 33, 250, 4111])
def test_pointwise_weight_gradient(ocnn, cin, cout, rows):
  torch.manual_seed(rows)
  x, g = torch.randn(1, cin, rows, 1, device='cuda'), torch.randn(1, cout, rows, 1, device='cuda')
  want = g.view(cout, rows).double() @ x.view(cin, rows).double().t()
  for nm in (False, True):
    xin = x.contiguous(memory_format=torch.channels_last) if nm else x
    assert off(ocnn.nn.pointwise_conv_weight_grad(xin, g), want) < 1e-6


def test_pointwise_training_layer(ocnn):
  """OctreeConv1x1 in training: every gradient, with and without a bias."""
  torch.manual_seed(5)
  for bias in (False, True):
    layer = ocnn.OctreeConv1x1(24, 64, bias).cuda().train()
    x = torch.randn(1, 24, 1000, 1, device='cuda', requires_grad=True)
    g = torch.randn(1, 64, 1000, 1, device='cuda')
    params = [x] + list(layer.parameters())
    got = torch.autograd.grad(layer(x), params, g)
    want = torch.autograd.grad(layer.conv1x1(x.squeeze(-1)).unsqueeze(-1), params, g)
    for a, b in zip(got, want):
      assert a.shape == b.shape and off(a, b.double()) < 2e-3     # (torch's own may run in TF32)


@pytest.mark.parametrize('cout', [63, 64, 96, 128, 129])
def test_weight_gradient_of_a_pointwise_training_layer(ocnn, cout):
  """The layer alone and in its block follow one rule, and inside it the weight gradient is fp32 throughout."""
  torch.manual_seed(cout)
  x, g = torch.randn(1, 32, 3000, 1, device='cuda'), torch.randn(1, cout, 3000, 1, device='cuda')
  layer, block = ocnn.OctreeConv1x1(32, cout).cuda().train(), ocnn.OctreeConv1x1Bn(32, cout).cuda().train()
  own = ocnn.nn.own_pointwise_weight_grad(layer.conv1x1.weight, x)
  assert own == (64 <= cout <= 128)
  assert not ocnn.nn.own_pointwise_weight_grad(layer.conv1x1.weight, x.half())
  assert not ocnn.nn.own_pointwise_weight_grad(layer.conv1x1.weight, x.contiguous(memory_format=torch.channels_last))
  want = g.view(cout, -1).double() @ x.view(32, -1).double().t()
  got, = torch.autograd.grad(layer(x), layer.conv1x1.weight, g)
  assert off(got.view(cout, 32), want) < (1e-6 if own else 2e-3)
  # the block's gradient reaches its 1x1 layer through the BatchNorm: the same through the modules one by one
  weight, bn = block.conv1x1.conv1x1.weight, block.bn
  y = torch.einsum('oc,nchw->nohw', weight.detach()[:, :, 0].double(), x.double()).float().requires_grad_()
  gy, = torch.autograd.grad(bn(y), y, g)
  got, = torch.autograd.grad(block(x), weight, g)
  assert off(got.view(cout, 32), gy.view(cout, -1).double() @ x.view(32, -1).double().t()) < 5e-3


class _Geometry(ctypes.Structure):
  _fields_ = [(n, ctypes.c_int32) for n in ('transposed', 'stride', 'nempty', 'h_in', 'h_out')] + \
      [(n, ctypes.c_void_p) for n in ('neigh', 'child', 'ichild')]


@pytest.mark.parametrize('ks', [[3, 3, 3], [2, 2, 2], [3, 1, 1], [1, 1, 1]])
@pytest.mark.parametrize('stride,nempty', [(1, False), (1, True), (2, False), (2, True)])
def test_weight_gradient_without_a_workspace(ocnn, octree, ks, stride, nempty):
  """ocnn_octree_conv_weight_grad: the CUDA-core form that asks for no device memory, through the C interface."""
  tree, v = octree
  lib, d, m, c = ctypes.CDLL(ocnn.LIBRARY), 5, 20, 9
  lib.ocnn_last_error.restype = ctypes.c_char_p
  neigh, child = (ocnn.octree_property(tree, p, d).contiguous() for p in ('neigh', 'child'))
  ichild = torch.nonzero(child >= 0).flatten().int()
  h_in = int(v.nnum_nempty[d] if nempty else v.nnum[d])
  h_out = int(v.nnum[d]) // 8 if stride == 2 else h_in
  x, a = torch.randn(1, c, h_in, 1, device='cuda'), torch.randn(1, m, h_out, 1, device='cuda')
  col = ocnn.nn.octree2col(x, tree, d, ks, stride, nempty).flatten(0, 1).double()
  taps = ks[0] * ks[1] * ks[2]
  want = a.view(m, h_out).double() @ col.view(c * taps, h_out).t()
  geo = _Geometry(0, stride, nempty, h_in, h_out, neigh.data_ptr(), child.data_ptr(), ichild.data_ptr())
  ptr = lambda t: ctypes.c_void_p(t.data_ptr())
  for node_major in (0, 1):
    xa, aa = ((t.view(t.shape[1], -1).t() if node_major else t).contiguous() for t in (x, a))
    got = torch.full((m, c * taps), 7.0, device='cuda')
    status = lib.ocnn_octree_conv_weight_grad(ptr(aa), ptr(xa), ptr(got), ctypes.byref(geo), m, c, (ctypes.c_int * 3)(*ks),
                                              node_major, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert status == 0, lib.ocnn_last_error()
    assert off(got, want) < 1e-6


def test_extreme_values(ocnn, octree):
  """Values whose high part would round to infinity, and tiny ones, keep their fp32 result."""
  tree, v = octree
  h = int(v.nnum[5])
  rng = np.random.default_rng(3)
  scale = torch.tensor(10.0 ** rng.uniform(-30, 30, size=h), dtype=torch.float32, device='cuda')
  x = torch.randn(1, 40, h, 1, device='cuda') * scale.view(1, 1, h, 1)
  x[0, 0, :4, 0] = torch.tensor([3.4e38, -3.4e38, 1e-40, 0.0], device='cuda')
  w = torch.zeros(32, 40 * 27, device='cuda')
  w[:, 13::27] = torch.randn(32, 40, device='cuda') * 1e-4      # the centre tap: a 1x1 layer
  got = ocnn.octree_conv(x, w, tree, 5, 32, [3, 3, 3], 1)
  want = (w[:, 13::27].double() @ x.view(40, h).double()).view(1, 32, h, 1)
  mag = (w[:, 13::27].double().abs() @ x.view(40, h).double().abs()).view(1, 32, h, 1)
  assert float(((got.double() - want).abs() / (mag + 1e-36)).max()) < 1e-6


def same_kinds(got, want):
  """Infinities of the same sign and NaNs in the same places, the rest finite and close."""
  finite = torch.isfinite(want)
  assert torch.equal(torch.isnan(got), torch.isnan(want))
  assert torch.equal(torch.isposinf(got), torch.isposinf(want)) and torch.equal(torch.isneginf(got), torch.isneginf(want))
  assert 0 < int(finite.sum()) < finite.numel()
  assert off(got[finite], want[finite].double()) < 2e-6


# (one and four weight images a stage, K splits and none; weights that bf16 holds exactly, whose lower parts
# are 0, and others, whose lower parts have either sign)
@pytest.mark.parametrize('cin,cout', [(40, 32), (64, 96)])
@pytest.mark.parametrize('depth', [5, 2])
@pytest.mark.parametrize('exact', [True, False])
def test_infinities(ocnn, octree, cin, cout, depth, exact):
  """An infinite operand gives what the chain of fp32 multiply-adds gives: forward, data and weight gradient."""
  tree, v = octree
  h = int(v.nnum[depth])
  torch.manual_seed(cin + depth)
  x, w = torch.randn(1, cin, h, 1, device='cuda'), torch.randn(cout, cin * 27, device='cuda') * 0.1
  g = torch.randn(1, cout, h, 1, device='cuda')
  if exact:
    x, w, g = (t.bfloat16().float() for t in (x, w, g))
  x[0, 0, 3, 0], x[0, 5, 70, 0], x[0, 7, 71, 0] = float('inf'), -float('inf'), float('inf')
  same_kinds(ocnn.nn.octree_conv(x, w, tree, depth, cout, [3, 3, 3], 1, False),
             ocnn.nn.octree_conv(x, w, tree, depth, cout, [3, 3, 3], 1, False, True))
  col = columns(ocnn, x, tree, depth, False)
  same_kinds(ocnn.nn.octree_conv_grad(x, w, tree, g, depth, cout, [3, 3, 3], 1, False, False, True)[1], g.view(cout, h).double() @ col.t())
  same_kinds(ocnn.nn.pointwise_conv(x, w[:, :cin].contiguous(), None, None, None, False),
             (w[:, :cin].double() @ x.view(cin, h).double()).view(1, cout, h, 1))
  g[0, 2, 9, 0] = -float('inf')
  x = x.nan_to_num(posinf=1.0, neginf=1.0)
  col = columns(ocnn, x, tree, depth, False)
  same_kinds(ocnn.nn.octree_conv_grad(x, w, tree, g, depth, cout, [3, 3, 3], 1, False, False, True)[1], g.view(cout, h).double() @ col.t())
  same_kinds(ocnn.nn.octree_deconv(g, w, tree, depth, cin, [3, 3, 3], 1, False),
             ocnn.nn.octree_deconv(g, w, tree, depth, cin, [3, 3, 3], 1, False, True))


@pytest.mark.parametrize('big', [False, True])
def test_which_kernel_a_training_layer_takes(ocnn, octree, big_octree, big):
  """Below 4 GFLOP forward and data gradient are the CUDA cores' chain bit for bit (ocnn_octree_conv_general), above
  it the tensor-core kernel's values."""
  tree, v = big_octree if big else octree
  d, c = (6, 64) if big else (5, 32)
  h = int(v.nnum[d])
  assert (2 * 27 * c * c * h > 4e9) == big
  layer = ocnn.OctreeConv(d, c, c).cuda().train()
  w = layer.weights.detach()
  x = torch.randn(1, c, h, 1, device='cuda', requires_grad=True)
  g = torch.randn(1, c, h, 1, device='cuda')
  y = layer(x, tree)
  gx, = torch.autograd.grad(y, x, g)
  if big:
    want = (ocnn.nn.octree_conv(x.detach(), w, tree, d, c, [3, 3, 3], 1, False),
            ocnn.nn.octree_deconv(g, w, tree, d, c, [3, 3, 3], 1, False))
  else:
    lib, neigh, want = ctypes.CDLL(ocnn.LIBRARY), ocnn.octree_property(tree, 'neigh', d).contiguous(), []
    for transposed, data in ((0, x.detach()), (1, g)):
      geo, out = _Geometry(transposed, 1, 0, h, h, neigh.data_ptr(), None, None), torch.empty_like(data)
      assert lib.ocnn_octree_conv_general(*(ctypes.c_void_p(t.data_ptr()) for t in (data, w, out)), ctypes.byref(geo), c, c,
                                          (ctypes.c_int * 3)(3, 3, 3), 0, 0, None,
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
      want.append(out)
  assert torch.equal(y.detach(), want[0]) and torch.equal(gx, want[1])


@pytest.mark.parametrize('shift', [0, 1, 2])
@pytest.mark.parametrize('cout', [32, 96])
def test_output_on_any_float_boundary(ocnn, octree, shift, cout):
  """ocnn_octree_conv_f32 writes node-major rows of whole float4 also where they are not aligned as such."""
  tree, v = octree
  d, cin, h = 5, 40, int(v.nnum[5])
  lib, ks = ctypes.CDLL(ocnn.LIBRARY), (ctypes.c_int * 3)(3, 3, 3)
  lib.ocnn_octree_conv_f32_workspace_bytes.restype = ctypes.c_size_t
  neigh = ocnn.octree_property(tree, 'neigh', d).contiguous()
  x, w = torch.randn(1, cin, h, 1, device='cuda'), torch.randn(cout, cin * 27, device='cuda') * 0.1
  rows = x.contiguous(memory_format=torch.channels_last)
  geo = _Geometry(0, 1, 0, h, h, neigh.data_ptr(), None, None)
  bytes_ = lib.ocnn_octree_conv_f32_workspace_bytes(ctypes.byref(geo), cin, cout, ks)
  ws, status = torch.empty(bytes_, dtype=torch.uint8, device='cuda'), torch.zeros(1, dtype=torch.int32, device='cuda')
  out = torch.full((h * cout + 8,), 5.0, device='cuda')
  ptr = lambda t: ctypes.c_void_p(t.data_ptr())
  assert lib.ocnn_octree_conv_f32(ptr(rows), ptr(w), ptr(out[shift:]), ctypes.byref(geo), cin, cout, ks, 1, None, ptr(ws),
                                  ctypes.c_size_t(bytes_), ptr(status),
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
  want = ocnn.octree_conv(rows, w, tree, d, cout, [3, 3, 3], 1)
  assert torch.equal(out[shift:shift + h * cout].view(h, cout).t(), want.view(cout, h))
  assert bool((out[:shift] == 5.0).all()) and bool((out[shift + h * cout:] == 5.0).all()) and int(status) == 0


@pytest.mark.parametrize('cout', [12800, 16000, 30000])
def test_very_many_output_channels(ocnn, octree, cout):
  """Where the epilogue's vectors leave no room for the ring the layer runs on the CUDA cores, as it did."""
  tree, v = octree
  h = int(v.nnum[2])
  x, w = torch.randn(1, 8, h, 1, device='cuda'), torch.randn(cout, 8 * 27, device='cuda') * 0.1
  want = (w.double() @ columns(ocnn, x, tree, 2, False)).view(1, cout, h, 1)
  assert off(ocnn.octree_conv(x, w, tree, 2, cout, [3, 3, 3], 1), want) < 2e-6
