"""Points buffers and octrees that are byte-wise views into other CUDA tensors: copied to a boundary where the call
takes them at all, refused with a message where it does not."""
import numpy as np
import pytest
import torch

import gpu_util as gu
from oracle import oracle as oc
from ocnn_harness import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ocnn():
  import ocnn as mod
  mod.set_key_bits(64)
  return mod


def shifted(t, by):
  big = torch.zeros(t.numel() + by, dtype=torch.uint8, device='cuda')
  big[by:] = t.cuda()
  return big[by:]


@pytest.mark.parametrize('by', [1, 2, 4])
@pytest.mark.parametrize('radius', [-1.0, 1.0])
def test_points(ocnn, by, radius):
  pts = torch.from_numpy(oc.points_new(*synth.primitive_union(3000, 1)))
  transform = ocnn.TransformCompose(dict(depth=5, full_depth=2, distort=False, radius=radius, center=(0.0, 0.0, 0.0)))
  for k, want in transform(pts).items():
    assert torch.equal(transform(shifted(pts, by))[k], want), k
  box = ocnn.bounding_sphere(shifted(pts, by), 'box')
  assert box == ocnn.bounding_sphere(pts, 'box')
  for a, b in zip(ocnn.clip_points(shifted(pts, by), [-0.5] * 3, [0.5] * 3), ocnn.clip_points(pts, [-0.5] * 3, [0.5] * 3)):
    assert torch.equal(a, b)


@pytest.mark.parametrize('by', [1, 4])
def test_octrees(ocnn, by):
  singles, merged, _ = gu.oracle_batch(gu.small_clouds(2, 2000, 300), 4, 2, 64)
  views = [shifted(torch.from_numpy(np.ascontiguousarray(o)), by) for o in singles]
  assert np.array_equal(ocnn.octree_batch(views).cpu().numpy(), merged)
  tree = shifted(torch.from_numpy(merged), by)
  x = torch.randn(1, 4, int(oc.OctreeView(merged).nnum[4]), 1, device='cuda')
  w = torch.randn(4, 4 * 27, device='cuda')
  pts = torch.zeros(5, 4, device='cuda')
  if by == 4:
    got = ocnn.octree_conv(x, w, tree, 4, 4, [3, 3, 3], 1)
    assert torch.equal(got, ocnn.octree_conv(x, w, gu.to_cuda_u8(merged), 4, 4, [3, 3, 3], 1))
    with pytest.raises(RuntimeError, match='boundary'):
      ocnn.nn.octree_interp(x, tree, 4, pts, 'nearest', False)
  else:
    with pytest.raises(RuntimeError, match='boundary'):
      ocnn.octree_conv(x, w, tree, 4, 4, [3, 3, 3], 1)
