"""The one-call preparation of a cloud behind TransformCompose against the four calls it stands for, bit for
bit: clouds that are clipped in part, entirely and not at all, host and device inputs, every property."""
import numpy as np
import pytest
import torch

from oracle import oracle as oc
from ocnn_harness import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ocnn():
  import ocnn as mod
  mod.set_key_bits(64)
  return mod


def cloud(n, seed, channels, labels):
  rng = np.random.default_rng(seed)
  p, q = synth.primitive_union(max(n, 8), seed)
  return torch.from_numpy(oc.points_new(
      p[:n] * 3 + 1, q[:n] if channels != 1 else None,
      rng.normal(size=(n, channels)).astype(np.float32) if channels else None,
      rng.integers(0, 5, size=n).astype(np.float32) if labels else None))


@pytest.mark.parametrize('n', [1, 255, 2048, 2049, 30001])
@pytest.mark.parametrize('channels,labels', [(0, False), (1, False), (3, True)])
@pytest.mark.parametrize('radius,center', [(-1.0, (-1.0,)), (1.5, (1.0, 1.2, 0.7)), (0.1, (50.0, 0.0, 0.0))])
def test_matches_the_separate_calls(ocnn, n, channels, labels, radius, center):
  pts = cloud(n, 3 + n, channels, labels)
  flags = dict(depth=5, full_depth=2, distort=True, offset=0.016, normal_axis='y', radius=radius, center=center)
  one = ocnn.TransformCompose(flags)

  class Points2Octree(ocnn.Points2Octree):      # (another class: call by call)
    pass
  each = ocnn.TransformCompose(flags)
  each.points2octree = Points2Octree(**flags)
  for src in (pts, pts.cuda()):
    np.random.seed(n)
    a = one(src)
    np.random.seed(n)
    b = each(src)
    for k in ('octree', 'points', 'inbox_mask'):
      assert a[k].is_cuda and torch.equal(a[k], b[k]), k
  assert torch.equal(pts, cloud(n, 3 + n, channels, labels))      # the input is left alone
