"""Where the batch builder changes its path: clouds at the sizes of a sort chunk, more clouds than ride
in the launch parameters, every digit width and key width, signals averaged into compact arrays (up
to six channels) or per node, bit-identical to the CPU oracle."""
import numpy as np
import pytest
import torch

import gpu_util as gu
from oracle import oracle as oc
from ocnn_harness import synth

pytestmark = pytest.mark.gpu
FLAGS = (False, False, False, False, 4, 0.1, 2.0, False, False, False)


@pytest.fixture(scope='module')
def ocnn():
  import ocnn as mod
  yield mod
  mod.set_key_bits(64)


def clouds_of(sizes, seed, channels=0, normals=True):
  rng = np.random.default_rng(seed)
  out = []
  for i, n in enumerate(sizes):
    p, q = synth.primitive_union(max(n, 8), seed + i)
    f = rng.normal(size=(n, channels)).astype(np.float32) if channels else None
    out.append(oc.points_new(p[:n], q[:n] if normals else None, f))
  return out


def check(ocnn, pts, depth, full, key_bits):
  ocnn.set_key_bits(key_bits)
  want = oc.octree_batch([oc.points2octree(p, depth, full, key_bits=key_bits) for p in pts])
  got = ocnn.points2octree_batch([torch.from_numpy(p) for p in pts], depth, full, *FLAGS).cpu().numpy()
  assert got.shape == want.shape and np.array_equal(got, want)


@pytest.mark.parametrize('depth,full,key_bits', [(1, 1, 64), (2, 1, 32), (2, 2, 64), (3, 1, 32), (5, 2, 64), (6, 2, 32), (6, 4, 64), (7, 2, 64),
                                                 (8, 2, 32), (9, 2, 64), (10, 3, 64), (11, 2, 64)])
def test_chunk_sizes(ocnn, depth, full, key_bits):
  check(ocnn, clouds_of([1, 2047, 2048, 2049, 4097, 700], 40 + depth), depth, full, key_bits)


@pytest.mark.parametrize('batch', [62, 63, 64, 150])
def test_many_small_clouds(ocnn, batch):
  rng = np.random.default_rng(batch)
  check(ocnn, clouds_of(rng.integers(1, 60, size=batch).tolist(), 900), 5, 2, 64)


@pytest.mark.parametrize('channels,normals', [(1, False), (6, False), (7, False), (3, True), (4, True)])
@pytest.mark.parametrize('depth', [5, 11])
def test_signal_channels(ocnn, channels, normals, depth):
  check(ocnn, clouds_of([1500, 900, 2500], 70, channels, normals), depth, 2, 64)


def test_several_tiles_per_chunk(ocnn):
  """Enough points that a sort chunk is more than one tile, in clouds that do not divide it."""
  check(ocnn, clouds_of([700000, 3, 600001], 11), 7, 2, 64)


@pytest.mark.parametrize('depth,key_bits,sizes', [
    # as many clouds as are sorted one by one whatever their size, and one more; a chunk of 2048 points that
    # holds a few clouds, hundreds, or the end of a large one; 32- and 64-bit composite keys, 8- and 9-bit digits
    (5, 64, [5] * 64), (5, 64, [5] * 65), (1, 64, [1] * 300), (3, 64, [3] * 1000), (8, 64, [9] * 70),
    (6, 32, [17, 1, 300] * 40), (9, 64, [40] * 500), (11, 64, [4000] + [2] * 200 + [2500, 1]),
    (6, 64, [7] * 5000)])
def test_batches_sorted_over_their_cloud_bits(ocnn, depth, key_bits, sizes):
  check(ocnn, clouds_of(sizes, 300), depth, min(depth, 2), key_bits)


@pytest.mark.parametrize('points', [6999, 7000])
def test_average_size_at_which_clouds_are_sorted_one_by_one(ocnn, points):
  check(ocnn, clouds_of([points - 500, points + 500] * 33, 77, channels=2), 6, 2, 64)
