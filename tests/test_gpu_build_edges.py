"""Where the batch builder changes its path: clouds at the sizes of a sort chunk, more clouds than ride
in the launch parameters, every digit width and key width, signals averaged into compact arrays (up
to six channels) or per node, bit-identical to the CPU oracle."""
import ctypes

import numpy as np
import pytest
import torch

import gpu_util as gu
from oracle import oracle as oc
from ocnn_harness import synth
from test_capi_host import Meta

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


class _Params(ctypes.Structure):
  _fields_ = [(n, ctypes.c_int32) for n in ('depth', 'full_depth', 'key_bits', 'merged', 'node_dis', 'split_label', 'save_pts',
                                            'adp_depth')] + \
      [('th_normal', ctypes.c_float), ('th_distance', ctypes.c_float), ('bbmin', ctypes.c_float * 3), ('bbmax', ctypes.c_float * 3)]


class _Batch(ctypes.Structure):
  _fields_ = [('batch', ctypes.c_int32), ('offsets', ctypes.c_void_p), ('xyz', ctypes.c_void_p), ('normal', ctypes.c_void_p),
              ('feature', ctypes.c_void_p), ('channels', ctypes.c_int32), ('label', ctypes.c_void_p)]


@pytest.mark.parametrize('shift', [0, 8, 16])
@pytest.mark.parametrize('depth', [5, 9, 11])              # (two and three sort passes, 32- and 64-bit keys)
def test_workspace_on_an_8_byte_boundary(ocnn, depth, shift):
  ocnn.set_key_bits(64)
  p, q = synth.primitive_union(7001, 5)
  want = oc.points2octree(oc.points_new(p, q), depth, 2, key_bits=64)
  xyz, nrm = torch.from_numpy(p).cuda(), torch.from_numpy(q).cuda()
  lib, meta = ctypes.CDLL(ocnn.LIBRARY), Meta()
  lib.ocnn_octree_build_workspace_bytes.restype = ctypes.c_size_t
  lib.ocnn_last_error.restype = ctypes.c_char_p
  size = lib.ocnn_octree_build_workspace_bytes(ctypes.c_int64(len(p)), 1, depth, 2)
  ws = torch.empty(size + 64, dtype=torch.uint8, device='cuda')
  offsets = (ctypes.c_int32 * 2)(0, len(p))
  xs, ns = (ctypes.c_void_p * 1)(xyz.data_ptr()), (ctypes.c_void_p * 1)(nrm.data_ptr())
  at = lambda a: ctypes.cast(a, ctypes.c_void_p)
  batch = _Batch(1, at(offsets), at(xs), at(ns), None, 0, None)
  params = _Params(depth, 2, 64, 0, 0, 0, 0, 4, 0.1, 2.0, (ctypes.c_float * 3)(-1, -1, -1), (ctypes.c_float * 3)(1, 1, 1))
  work, stream = ctypes.c_void_p(ws.data_ptr() + shift), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
  assert lib.ocnn_octree_build_plan(ctypes.byref(batch), ctypes.byref(params), work, ctypes.c_size_t(size), ctypes.byref(meta),
                                    stream) == 0, lib.ocnn_last_error()
  out = torch.empty(meta.ptr_dis[6], dtype=torch.uint8, device='cuda')
  assert lib.ocnn_octree_build_emit(ctypes.byref(batch), ctypes.byref(params), ctypes.byref(meta), work, ctypes.c_size_t(size),
                                    ctypes.c_void_p(out.data_ptr()), ctypes.c_size_t(out.numel()), None, stream) == 0
  torch.cuda.synchronize()
  assert np.array_equal(out.cpu().numpy(), want)


# One cloud of up to 6144 points is sorted by one launch, others by several: the edges of each, a single point, rows that do not fill up, every
# number of passes; and the chunk edges of the longer way.
@pytest.mark.parametrize('sizes', [[1], [33], [1024], [1025], [6143], [6144], [6145], [1, 2047, 2048]])
@pytest.mark.parametrize('depth,full,key_bits', [(1, 1, 64), (5, 2, 64), (6, 2, 32), (8, 2, 64), (9, 2, 64), (10, 1, 64)])
def test_one_launch_or_several(ocnn, sizes, depth, full, key_bits):
  check(ocnn, clouds_of(sizes, 300 + sum(sizes)), depth, full, key_bits)


def test_points_in_one_cell(ocnn):
  p = np.full((3000, 3), 0.123, np.float32)
  q = np.tile(np.float32([0, 0, 1]), (3000, 1))
  check(ocnn, [oc.points_new(p, q)], 6, 2, 64)
