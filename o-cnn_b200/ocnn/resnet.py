"""The reference's classification ResNet (pytorch/ocnn/resnet.py:5-31): a 3x3x3 stem at `depth`,
then per level d = depth .. 3 `resblk_num` bottleneck blocks and a max-pool, channels
2^max(11 - d, 2), a global average over the full level 2 and one linear layer."""
import torch
from torch import nn as _nn

from . import nn
from .modules import OctreeConvBnRelu, OctreeResBlocks, hooked
from .octree2voxel import FullOctree2Voxel
from .octree_pool import OctreeMaxPool, FullOctreeGlobalPool


class ResNet(_nn.Module):
  def __init__(self, depth, channel_in, nout, resblk_num):
    super().__init__()
    self.depth, self.channel_in = depth, channel_in
    width = lambda d: 2 ** max(11 - d, 2)
    self.conv1 = OctreeConvBnRelu(depth, channel_in, width(depth))
    levels = range(depth, 2, -1)
    self.resblocks = _nn.ModuleList(
        OctreeResBlocks(d, width(min(d + 1, depth)), width(d), resblk_num) for d in levels)
    self.pools = _nn.ModuleList(OctreeMaxPool(d) for d in levels)
    self.header = _nn.Sequential(FullOctreeGlobalPool(depth=2), _nn.Linear(width(3), nout))

  def forward(self, octree, data=None):
    """`data` overrides the octree's stored signal (e.g. a bfloat16 channels_last copy of it)."""
    if data is None:
      data = nn.octree_property(octree, 'feature', self.depth)
    assert data.size(1) == self.channel_in
    data = self.conv1(data, octree)
    for blocks, pool in zip(self.resblocks, self.pools):
      data = pool(blocks(data, octree), octree)
    if self._head_is_one_kernel(data):
      pool, fc = self.header
      return nn.global_pool_fc(data, fc.weight, fc.bias, data.shape[2] // 8 ** pool.depth)
    return self.header(data.float() if data.dtype != torch.float32 else data)

  def _head_is_one_kernel(self, data):
    """Whether the header can run as pool + Linear in one launch: the two stock modules with nothing that
    would have to see the tensors between them, on 16-bit node-major data, with no gradient to record
    (a frozen network whose Linear is being trained records one)."""
    if self.training or data.dtype not in (torch.bfloat16, torch.float16) or torch.is_autocast_enabled():
      return False
    head = self.header
    if type(head) is not _nn.Sequential or len(head._modules) != 2:
      return False
    pool, fc = head._modules.values()
    if type(pool) is not FullOctreeGlobalPool or type(fc) is not _nn.Linear:
      return False
    voxel = pool.octree2voxel
    if type(voxel) is not FullOctree2Voxel or hooked(head, pool, voxel, fc):
      return False
    weight, bias = fc.weight, fc.bias
    if weight.dtype != torch.float32 or (bias is not None and bias.dtype != torch.float32) or \
        not data.is_contiguous(memory_format=torch.channels_last):
      return False
    return not (torch.is_grad_enabled() and (data.requires_grad or weight.requires_grad or
                                             (bias is not None and bias.requires_grad)))
