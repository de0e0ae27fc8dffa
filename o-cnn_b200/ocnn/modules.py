"""Building blocks of the reference's networks (pytorch/ocnn/modules.py:1-345):
convolution + BatchNorm (+ ReLU) blocks, 1x1 blocks, the two residual blocks, nearest /
trilinear interpolation at points, and `octree_feature`.  Class names, constructor arguments and
parameter names follow the reference, so its state_dicts load.

In eval mode a block folds its BatchNorm (running statistics) and ReLU into the convolution
kernel's epilogue — one launch per block instead of three; set `FUSE_EVAL_BN = False` to run the
torch BatchNorm / ReLU modules after the convolution instead.  In training mode an fp32 block is one
native autograd node around the same convolution kernel and torch's own BatchNorm (`_train_block`);
under autocast, with hooks on the inner modules, or with another normalisation the modules run one
by one.
"""
import torch
from torch import nn as _nn
from torch.autograd import forward_ad

from . import nn
from .octree_conv import OctreeConv, OctreeDeconv, bn_vectors, tc_status
from .octree_pool import OctreeMaxPool
from .octree_pad import octree_depad
from .octree_pad import OctreeTile  # noqa: F401  (re-exported: the reference defines it here)

bn_momentum, bn_eps = 0.01, 0.001       # pytorch/ocnn/modules.py:5
FUSE_EVAL_BN = True


def _trainable(data, weight, bn, residual, *passed_by):
  """Whether a block in training mode can run as the one native autograd node: plain fp32 on the GPU,
  a BatchNorm with parameters and running statistics, no hooks that would have to see it or the other modules
  passed by."""
  return (torch.is_grad_enabled() and bn.training and data.is_cuda and data.dtype == torch.float32 and
          data.is_contiguous() and weight.dtype == torch.float32 and weight.is_cuda and bn.affine and
          bn.track_running_stats and bn.momentum is not None and bn._parameters['weight'].dtype == torch.float32 and
          (residual is None or residual.dtype == torch.float32) and not torch.is_autocast_enabled() and
          not hooked(bn, *passed_by) and _only_backward())


def hooked(*modules):
  """Whether someone asked to see these modules' calls: a path that passes them by has to leave them alone."""
  for m in modules:
    if m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks:
      return True
  return bool(torch.nn.modules.module._has_any_global_hook())


_functorch_level = torch._C._functorch.peek_interpreter_stack
_tracing_state, _compiling = torch._C._get_tracing_state, torch.compiler.is_compiling


def _only_backward():
  """Whether no more than reverse-mode autograd looks on: a functorch transform, a level of forward-mode
  derivatives, a tracer or a compiler has to see torch's own operators."""
  return (_functorch_level() is None and forward_ad._current_level < 0 and _tracing_state() is None and
          not _compiling())


def _stock_conv1x1(conv):
  """Whether a 1x1 layer's product may be formed from the weight and bias of `conv` without calling it."""
  return (type(conv) is _nn.Conv1d and conv.kernel_size == (1,) and conv.stride == (1,) and
          conv.padding == (0,) and conv.groups == 1)


def _train_block(data, weight, bias, bn, residual, octree, kind, depth, cout, kernel_size, stride, nempty, relu):
  own, stats = bn._parameters, bn._buffers       # (Module's own look-up costs 0.4 us a name)
  return nn.train_block(data, weight, bias, own['weight'], own['bias'], residual, stats['running_mean'],
                        stats['running_var'], bn.momentum, bn.eps, octree, kind, depth, cout, kernel_size, stride,
                        nempty, relu, stats['num_batches_tracked'])


def _folded(bn):
  """(scale, bias) float32 vectors equal to an eval-mode BatchNorm."""
  with torch.no_grad():
    scale = bn.weight.float() / torch.sqrt(bn.running_var.float() + bn.eps)
    bias = bn.bias.float() - bn.running_mean.float() * scale
  return scale.contiguous(), bias.contiguous()


class _OctreeBlock(_nn.Module):
  """An octree (de)convolution followed by BatchNorm2d and optionally ReLU."""
  layer, attr, with_relu = OctreeConv, 'conv', True

  def __init__(self, depth, channel_in, channel_out, kernel_size=[3], stride=1, nempty=False):
    super().__init__()
    setattr(self, self.attr, self.layer(depth, channel_in, channel_out, kernel_size, stride, nempty))
    self.bn = _nn.BatchNorm2d(channel_out, bn_eps, bn_momentum)
    if self.with_relu:
      self.relu = _nn.ReLU(inplace=True)

  def forward(self, data_in, octree, residual=None, relu=None):
    op = getattr(self, self.attr)
    relu = self.with_relu if relu is None else relu
    # a stride-2 convolution on all nodes is padded AFTER the kernel, and BatchNorm must see the
    # padded zeros: it cannot be folded into the kernel there
    foldable = not (op.is_conv_layer() and op.stride == 2 and not op.nempty)
    if FUSE_EVAL_BN and foldable and not self.training:
      assert data_in.size(1) == op.channel_in
      if not op.is_conv_layer() and op.stride == 2 and not op.nempty:
        data_in = nn.octree_depad(data_in, octree, op.depth)
      return op._run(data_in, octree, self.bn, residual, relu)
    bn = self.bn
    if foldable and type(bn) is _nn.BatchNorm2d and type(op) in (OctreeConv, OctreeDeconv) and \
        _trainable(data_in, op.weights, bn, residual, op):
      assert data_in.size(1) == op.channel_in
      if not op.is_conv_layer() and op.stride == 2 and not op.nempty:
        data_in = octree_depad(data_in, octree, op.depth)
      return _train_block(data_in, op.weights, None, bn, residual, octree, int(not op.is_conv_layer()),
                          op.depth, op.channel_out, op.kernel_size, op.stride, op.nempty, relu)
    out = bn(op(data_in, octree))
    if residual is not None:
      out = out + residual
    return torch.relu_(out) if relu else out


class OctreeConvBn(_OctreeBlock):
  with_relu = False


class OctreeConvBnRelu(_OctreeBlock):
  pass


class OctreeDeConvBnRelu(_OctreeBlock):
  layer, attr = OctreeDeconv, 'deconv'


class FcBnRelu(_nn.Module):
  def __init__(self, channel_in, channel_out):
    super().__init__()
    self.flatten = _nn.Flatten(start_dim=1)
    self.fc = _nn.Linear(channel_in, channel_out, bias=False)
    self.bn = _nn.BatchNorm1d(channel_out, bn_eps, bn_momentum)
    self.relu = _nn.ReLU(inplace=True)

  def forward(self, data_in):
    return self.relu(self.bn(self.fc(self.flatten(data_in))))


class _Conv1x1Function(torch.autograd.Function):
  """torch's own 1x1 convolution with this library's kernel for the weight gradient (torch's where that is to be
  differentiated again)."""

  @staticmethod
  def forward(ctx, data, weight, bias):
    ctx.save_for_backward(data, weight)
    ctx.bias = None if bias is None else list(bias.shape)
    return torch.conv1d(data.squeeze(-1), weight, bias).unsqueeze(-1)

  @staticmethod
  def backward(ctx, grad):
    data, weight = ctx.saved_tensors
    need_x, need_w, need_b = ctx.needs_input_grad
    grad = grad.contiguous()
    gx = gw = gb = None
    own = need_w and not torch.is_grad_enabled()
    if need_x or need_b or (need_w and not own):
      gx, gw, gb = torch.ops.aten.convolution_backward(
          grad.squeeze(-1), data.squeeze(-1), weight, ctx.bias, [1], [0], [1], False, [0], 1,
          [need_x, need_w and not own, need_b])
      gx = gx if gx is None else gx.unsqueeze(-1)
    if own:
      gw = nn.pointwise_conv_weight_grad(data, grad).view_as(weight)
    return gx, gw, gb


class OctreeConv1x1(_nn.Module):
  """A per-node linear map.  The parameters live in a torch Conv1d (as in the reference, so the
  state_dict keys match); the product runs on this library's pointwise kernels."""
  _layer = None

  def __init__(self, channel_in, channel_out, use_bias=False):
    super().__init__()
    self.conv1x1 = _nn.Conv1d(channel_in, channel_out, kernel_size=1, bias=use_bias)

  def run(self, data_in, bn=None, residual=None, relu=False):
    """The product, and the BatchNorm on its running statistics, residual and ReLU that follow it."""
    conv = self.conv1x1
    if torch.is_grad_enabled() and (data_in.requires_grad or
                                    (self.training and conv.weight.requires_grad)):
      # training: torch's own 1x1 convolution (as the reference), which autograd differentiates; for some
      # widths with this library's weight gradient
      if nn.own_pointwise_weight_grad(conv.weight, data_in) and not torch.is_autocast_enabled() and \
          _stock_conv1x1(conv) and not hooked(conv) and _only_backward():
        out = _Conv1x1Function.apply(data_in, conv.weight, conv.bias)
      else:
        out = conv(data_in.squeeze(-1)).unsqueeze(-1)
      if bn is not None:
        scale, bias = _folded(bn)
        out = out * scale.view(1, -1, 1, 1) + bias.view(1, -1, 1, 1)
      if residual is not None:
        out = out + residual
      return torch.relu(out) if relu else out
    if self._layer is None:
      cout, cin = conv.weight.shape[:2]
      self._layer = nn.ConvLayer(cin, cout, [1, 1, 1], 1, False, False, True)
    affine = bn_vectors(bn)
    if conv.bias is not None:
      with torch.no_grad():
        b = conv.bias.detach().float()
        if bn is None:
          affine = (None, b, None, None, 0.0)
        else:
          scale, bias = _folded(bn)
          affine = (scale, bias + b * scale, None, None, 0.0)
    return self._layer.run(data_in, conv.weight, None, 0, *affine, residual, relu,
                           tc_status(data_in.device))

  def forward(self, data_in):
    return self.run(data_in)


class _Conv1x1Block(_nn.Module):
  with_relu = True

  def __init__(self, channel_in, channel_out, use_bias=False):
    super().__init__()
    self.conv1x1 = OctreeConv1x1(channel_in, channel_out, use_bias)
    self.bn = _nn.BatchNorm2d(channel_out, bn_eps, bn_momentum)
    if self.with_relu:
      self.relu = _nn.ReLU(inplace=True)

  def forward(self, data_in, residual=None, relu=None):
    relu = self.with_relu if relu is None else relu
    if FUSE_EVAL_BN and not self.training:
      return self.conv1x1.run(data_in, self.bn, residual, relu)
    layer, bn = self.conv1x1, self.bn
    conv = layer.conv1x1
    if type(bn) is _nn.BatchNorm2d and type(layer) is OctreeConv1x1 and _stock_conv1x1(conv):
      weight = conv.weight
      if _trainable(data_in, weight, bn, residual, conv, layer):
        return _train_block(data_in, weight, conv.bias, bn, residual, None, 2, 0, weight.shape[0], [1], 1, False, relu)
    out = bn(layer(data_in))
    if residual is not None:
      out = out + residual
    return torch.relu_(out) if relu else out


class OctreeConv1x1Bn(_Conv1x1Block):
  with_relu = False


class OctreeConv1x1BnRelu(_Conv1x1Block):
  pass


class _ResBlockBase(_nn.Module):
  def __init__(self, depth, channel_in, channel_out, stride, nempty):
    super().__init__()
    self.channel_in, self.channel_out = channel_in, channel_out
    self.stride, self.depth = stride, depth
    if stride == 2:
      self.maxpool = OctreeMaxPool(depth)
      self.depth = depth - 1
    self.relu = _nn.ReLU(inplace=True)

  def _finish(self, last, branch, skip_proj, data_in, *octree):
    """relu(last(branch) + skip): in eval mode the sum and the ReLU ride in `last`'s epilogue."""
    skip = data_in if skip_proj is None else skip_proj(data_in)
    return last(branch, *octree, residual=skip, relu=True)


class OctreeResBlock(_ResBlockBase):
  """Bottleneck: 1x1 -> 3x3x3 at channel_out / bottleneck -> 1x1, plus the (projected) input."""

  def __init__(self, depth, channel_in, channel_out, stride=1, bottleneck=4, nempty=False):
    super().__init__(depth, channel_in, channel_out, stride, nempty)
    self.bottleneck = bottleneck
    channelb = int(channel_out / bottleneck)
    self.conv1x1a = OctreeConv1x1BnRelu(channel_in, channelb)
    self.conv3x3 = OctreeConvBnRelu(self.depth, channelb, channelb, nempty=nempty)
    self.conv1x1b = OctreeConv1x1Bn(channelb, channel_out)
    if channel_in != channel_out:
      self.conv1x1c = OctreeConv1x1Bn(channel_in, channel_out)

  def forward(self, data_in, octree):
    if self.stride == 2:
      data_in = self.maxpool(data_in, octree)
    mid = self.conv3x3(self.conv1x1a(data_in), octree)
    proj = self.conv1x1c if self.channel_in != self.channel_out else None
    return self._finish(self.conv1x1b, mid, proj, data_in)


class OctreeResBlock2(_ResBlockBase):
  """Two 3x3x3 convolutions, plus the (projected) input."""

  def __init__(self, depth, channel_in, channel_out, stride=1, bottleneck=1, nempty=False):
    super().__init__(depth, channel_in, channel_out, stride, nempty)
    channelb = int(channel_out / bottleneck)
    self.conv3x3a = OctreeConvBnRelu(self.depth, channel_in, channelb, nempty=nempty)
    self.conv3x3b = OctreeConvBn(self.depth, channelb, channel_out, nempty=nempty)
    if channel_in != channel_out:
      self.conv1x1 = OctreeConv1x1Bn(channel_in, channel_out)

  def forward(self, data_in, octree):
    if self.stride == 2:
      data_in = self.maxpool(data_in, octree)
    mid = self.conv3x3a(data_in, octree)
    proj = self.conv1x1 if self.channel_in != self.channel_out else None
    return self._finish(self.conv3x3b, mid, proj, data_in, octree)


class OctreeResBlocks(_nn.Module):
  def __init__(self, depth, channel_in, channel_out, resblk_num, bottleneck=4, nempty=False,
               resblk=OctreeResBlock, use_checkpoint=False):
    super().__init__()
    self.resblk_num = resblk_num
    self.use_checkpoint = use_checkpoint       # training-time memory saving: no effect here
    widths = [channel_in] + [channel_out] * resblk_num
    self.resblks = _nn.ModuleList(
        resblk(depth, widths[i], widths[i + 1], 1, bottleneck, nempty) for i in range(resblk_num))

  def forward(self, data, octree):
    for blk in self.resblks:
      data = blk(data, octree)
    return data


def create_full_octree(depth, channel, batch_size=1, node_dis=True):
  """A full octree of the given depth, grown level by level from octree_new
  (pytorch/ocnn/modules.py:325-330)."""
  assert depth > 1
  octree = nn.octree_new(batch_size, channel, node_dis)
  for target_depth in range(1, depth + 1):
    octree = nn.octree_grow(octree, target_depth, full_octree=True)
  return octree


def octree_feature(octree, depth, nempty=False):
  """The octree's stored signal at `depth` as [1,C,H,1] (on the non-empty nodes when nempty)."""
  out = nn.octree_property(octree, 'feature', depth)
  return nn.octree_depad(out, octree, depth) if nempty else out


# ---- interpolation of node data at points (pytorch/ocnn/modules.py:209-316) -------------------------
def octree_nearest_pts(data, octree, depth, pts, nempty=False):
  """Rows of the cells holding the points.  pts: [N, 4] = (x, y, z) scaled to [0, 2^depth] and the
  batch id; returns [1, C, N, 1] (zeros for points in no cell)."""
  with torch.no_grad():
    return nn.octree_interp(data, octree, depth, pts, 'nearest', nempty)


def octree_trilinear_pts(data, octree, depth, pts, nempty=False):
  """Trilinear interpolation over the 8 cells around each point, renormalised over the cells that
  exist.  One kernel: key arithmetic, search and the weighted sum (the reference builds a sparse
  matrix and multiplies twice)."""
  with torch.no_grad():
    return nn.octree_interp(data, octree, depth, pts, 'linear', nempty)


def octree_trilinear(data, octree, depth, target_depth):
  """Interpolate data from level `depth` at the cell centres of level `target_depth`."""
  xyz = nn.octree_property(octree, 'xyz', target_depth)
  xyz = nn.octree_decode_key(xyz).float()
  scale = 2.0 ** (depth - target_depth)
  xyz = (xyz + xyz.new_tensor([0.5, 0.5, 0.5, 0.0])) * xyz.new_tensor([scale, scale, scale, 1.0])
  return octree_trilinear_pts(data, octree, depth, xyz)


class OctreeTrilinear(_nn.Module):
  def __init__(self, depth):
    super().__init__()
    self.depth = depth

  def forward(self, data, octree):
    return octree_trilinear(data, octree, self.depth, self.depth + 1)


class OctreeInterp(_nn.Module):
  def __init__(self, depth, method='linear', nempty=False):
    super().__init__()
    self.depth, self.method, self.nempty = depth, method, nempty

  def forward(self, data, octree, pts):
    # pts in [-1, 1] -> [0, 2^depth]
    xyz = (pts[:, :3] + 1.0) * (2 ** (self.depth - 1))
    pts = torch.cat([xyz, pts[:, 3:]], dim=1)
    if self.method == 'nearest':
      return octree_nearest_pts(data, octree, self.depth, pts, self.nempty)
    if self.method == 'linear':
      return octree_trilinear_pts(data, octree, self.depth, pts, self.nempty)
    raise ValueError(self.method)

  def extra_repr(self) -> str:
    return 'depth={}, method={}, nempty={}'.format(self.depth, self.method, self.nempty)
