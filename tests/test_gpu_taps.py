"""Tap plans (`ocnn.nn.TapPlan`): the order and masks against numpy, and the convolution on a plan against the walk
over all taps, which it equals bit for bit where that one does not split K."""
import numpy as np
import pytest
import torch

import gpu_util as gu
from ocnn_harness import synth
from oracle import oracle as oc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ocnn():
  import ocnn as mod
  mod.set_key_bits(64)
  return mod


@pytest.fixture(scope='module')
def small():
  """Levels of 1 to about 3 k non-empty nodes."""
  _, merged, _ = gu.oracle_batch(gu.small_clouds(3, 3000, 500), 5, 2, 64)
  return gu.to_cuda_u8(merged), oc.OctreeView(merged)


@pytest.fixture(scope='module')
def large(ocnn):
  """About 97 k non-empty nodes at depth 7, a slab among scattered points: from 1 to 27 neighbours."""
  gen = torch.Generator().manual_seed(7)
  p = 0.99 * (2 * torch.rand(100000, 3, generator=gen) - 1)
  p[50000:] = p[50000:] * torch.tensor([1.0, 1.0, 0.02])
  n = torch.nn.functional.normalize(torch.randn(100000, 3, generator=gen), dim=1)
  return ocnn.octree_batch([ocnn.Points2Octree(7, 2)(ocnn.points_new(p, n, torch.zeros(0), torch.zeros(0)))]).cuda()


def neighbour_sets(ocnn, octree, d):
  """[rows, 27] which neighbours of a level's non-empty nodes are non-empty."""
  child = ocnn.octree_property(octree, 'child', d).cpu().numpy()
  neigh = ocnn.octree_property(octree, 'neigh', d).cpu().numpy().reshape(-1, 64)
  t = np.arange(27)
  h = np.nonzero(child >= 0)[0]
  code = ((h & 4) << 2) | ((h & 2) << 1) | (h & 1)
  at = neigh[h >> 3][np.arange(h.size)[:, None], ((t // 9 << 4) | (t // 3 % 3 << 2) | t % 3)[None] + code[:, None]]
  return (at >= 0) & (child[np.maximum(at, 0)] >= 0)


def check_plan(ocnn, octree, plan, d):
  sets = neighbour_sets(ocnn, octree, d)
  order, mask = (t.cpu().numpy() for t in plan.level(d))
  live = order >= 0
  assert np.array_equal(np.sort(order[live]), np.arange(len(sets))) and live[:len(sets)].all()
  per_row = (sets.astype(np.int64) << np.arange(27)).sum(1)
  want = np.where(live, per_row[np.maximum(order, 0)], 0).reshape(-1, 128)
  assert np.array_equal(np.bitwise_or.reduce(want, axis=1), mask)
  return sets, mask


def test_plan_of_all_levels(ocnn, small, large):
  octree, v = small
  plan = ocnn.nn.TapPlan(octree, [5, 4, 3, 2, 1, 0, 9])      # (levels that are not there are left out)
  for d in range(1, 6):
    check_plan(ocnn, octree, plan, d)
  with pytest.raises(RuntimeError):
    plan.level(0)
  plan = ocnn.nn.TapPlan(large, [7, 6, 5])
  for d in (7, 6, 5):
    sets, mask = check_plan(ocnn, large, plan, d)
  sets, mask = check_plan(ocnn, large, plan, 7)
  tile_taps = np.unpackbits(mask.view(np.uint8)).sum() / mask.size
  assert sets.sum(1).mean() <= tile_taps < 17                 # (in Morton order it is 27)


def wipe_neighbours(octree, d):
  """Neighbour table of a level set to "none", through memory that torch takes for another tensor's."""
  v = oc.OctreeView(octree.cpu().numpy())
  at = int(v.ptr_dis[oc.PROPS.index('neigh')]) + 32 * int(v.nnum_cum[d])
  torch.from_dlpack(octree)[at:at + 32 * int(v.nnum[d])] = 255


def both(ocnn, octree, d, cin, cout, dtype, with_res=False, edit=None):
  """The layer over all taps and on a plan.  A plan has its own tables: the layer runs on it after the octree's were
  wiped, which the walk over all taps does not survive."""
  h = int((ocnn.octree_property(octree, 'child', d) >= 0).sum())
  torch.manual_seed(cin + cout + d)
  fmt = dict(memory_format=torch.channels_last)
  x = torch.randn(1, cin, h, 1, device='cuda').to(dtype).contiguous(**fmt)
  res = torch.randn(1, cout, h, 1, device='cuda').to(dtype).contiguous(**fmt) if with_res else None
  bn = torch.nn.BatchNorm2d(cout).cuda().eval() if with_res else None
  layer = ocnn.OctreeConv(d, cin, cout, nempty=True).cuda().eval()
  if edit is not None:
    edit(layer.weights)
  base = octree.clone()
  planned = base.view(-1)
  planned.tap_plan = ocnn.nn.TapPlan(base, [d])
  with torch.no_grad():
    want = layer._run(x, base, bn, res, with_res)
    wipe_neighbours(base, d)
    assert not torch.equal(layer._run(x, base, bn, res, with_res), want)
    assert planned.tap_plan.serves(planned, d, h)
    return want, layer._run(x, planned, bn, res, with_res)


# (channels that share K-blocks between taps, that leave a remainder, that fill 1 to 8 blocks; output columns of
# one 16-column piece, with a remainder of 8, of one and of two slices)
@pytest.mark.parametrize('cin,cout', [(16, 8), (32, 32), (48, 40), (96, 96), (128, 96), (192, 128), (64, 256), (32, 512),
                                      (512, 16)])
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16])
@pytest.mark.parametrize('with_res', [False, True])
def test_convolution_on_a_plan(ocnn, small, large, cin, cout, dtype, with_res):
  for octree, d in ((large, 7), (small[0], 5), (small[0], 4), (small[0], 1)):
    a, b = both(ocnn, octree, d, cin, cout, dtype, with_res)
    if octree is large or cin <= 64:       # (fewer than 32 K-blocks, or tiles for every SM: K is not split)
      assert torch.equal(a, b)
    else:                                  # sums of parts: fp32 sums of up to 27 cin terms, rounded to 16 bits once
      ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
      assert bool(((a.float() - b.float()).abs() <= 2 * ulp * a.float().abs() + 1e-5 * float(a.float().abs().max())).all())


@pytest.mark.parametrize('value', [float('inf'), float('nan'), 1e6])     # (1e6: infinite as float16)
def test_weights_that_are_not_finite(ocnn, small, value):
  def edit(w):
    with torch.no_grad():
      w[3, 27 * 5 + 0] = value             # a corner tap: most tiles have none of it
  a, b = both(ocnn, small[0], 5, 32, 32, torch.float16, edit=edit)
  assert bool(torch.isnan(a).any())
  torch.testing.assert_close(a, b, rtol=0, atol=0, equal_nan=True)


def test_a_plan_serves_only_what_it_was_made_for(ocnn, small):
  octree = small[0].clone()
  h = int((ocnn.octree_property(octree, 'child', 5) >= 0).sum())
  # as many nodes on every level, others: the same clouds with x and y swapped
  _, swapped, _ = gu.oracle_batch([[a[:, [1, 0, 2]] for a in c[:2]] for c in gu.small_clouds(3, 3000, 500)], 5, 2, 64)
  swapped = gu.to_cuda_u8(swapped)
  assert ocnn.nn.octree_info(swapped) == ocnn.nn.octree_info(octree) and swapped.numel() == octree.numel()
  x = torch.randn(1, 32, h, 1, device='cuda').bfloat16().contiguous(memory_format=torch.channels_last)
  layer = ocnn.OctreeConv(5, 32, 32, nempty=True).cuda().eval()
  planned = octree.view(-1)
  plan = planned.tap_plan = ocnn.nn.TapPlan(octree, [5])
  with torch.no_grad():
    want, want_swapped = layer(x, octree), layer(x, swapped)
    assert not torch.equal(want, want_swapped)
    assert plan.serves(planned, 5, h) and plan.serves(octree, 5, h)
    assert not (plan.serves(planned, 4, h) or plan.serves(planned, 5, h - 1) or plan.serves(small[0], 5, h))
    assert torch.equal(layer(x, planned), want)
    other = torch.cuda.Stream()
    other.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(other):
      assert not plan.serves(planned, 5, h)                # made by work that this stream need not have waited for
      got = layer(x, planned)
    torch.cuda.current_stream().wait_stream(other)
    assert torch.equal(got, want)
    other_octree = swapped.view(-1)
    other_octree.tap_plan = plan
    assert torch.equal(layer(x, other_octree), want_swapped)
    planned.copy_(swapped)                 # written to since
    assert not plan.serves(planned, 5, h)
    assert torch.equal(layer(x, planned), want_swapped)


# ---- the network on its plans --------------------------------------------------------------------------------
@pytest.fixture(scope='module')
def scene(ocnn):
  """An octree whose levels 9 to 7 have more tiles than SMs and go on a plan, and whose levels 6 and 5 do not."""
  xyz, nrm, rgb = (torch.from_numpy(t) for t in synth.indoor_scene(120000, 11))
  octree = ocnn.Points2Octree(9, 2).batch([ocnn.points_new(xyz, nrm, rgb, torch.zeros(0))])
  rows = {d: int((ocnn.octree_property(octree, 'child', d) >= 0).sum()) for d in range(5, 10)}
  one_wave = 128 * torch.cuda.get_device_properties(0).multi_processor_count
  planned = {d for d in rows if rows[d] > one_wave}
  assert planned and set(rows) - planned and max(rows.values()) > 2 * one_wave, rows
  pts = torch.cat([xyz[:5000], torch.zeros(5000, 1)], 1).cuda()
  return octree, rows, planned, pts


def make_unet(ocnn, seed):
  torch.manual_seed(seed)
  net = ocnn.UNet(9, 8, 20, nempty=True).cuda()
  with torch.no_grad():
    for m in net.modules():
      if isinstance(m, (torch.nn.BatchNorm1d, torch.nn.BatchNorm2d)):
        m.weight.uniform_(0.5, 1.5), m.bias.uniform_(-0.2, 0.2)
        m.running_mean.uniform_(-0.2, 0.2), m.running_var.uniform_(0.5, 1.5)
  return net.eval()


def node_data(octree, ocnn, dtype):
  half = dtype == torch.float16
  return ocnn.octree_depad(ocnn.nn.feature_node_major(octree, 8, not half, half), octree, 9)


@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16])
def test_network_on_plans_is_the_network_without(ocnn, scene, dtype, monkeypatch):
  """`UNet.forward` with the plans it makes: every 3x3x3 layer of a larger level finds one (conv1, of 8 channels, does
  not take it) and the others do not, down and up again, and the scores are those of the walk over all taps bit for bit."""
  octree, rows, planned, pts = scene
  net, data = make_unet(ocnn, 5), node_data(octree, ocnn, dtype)
  base, make, seen = ocnn.OctreeConv.__base__, ocnn.unet._with_tap_plan, []
  run = base._run

  def spy(layer, x, o, *args):
    plan = getattr(o, 'tap_plan', None)
    seen.append((layer, x.shape[2], plan is not None and plan.serves(o, layer.depth, x.shape[2])))
    return run(layer, x, o, *args)

  with torch.no_grad():
    monkeypatch.setattr(ocnn.unet, '_with_tap_plan', lambda o, depths, x: o)
    want, want_nodes = net(octree, pts, data), net(octree, None, data)
    monkeypatch.setattr(ocnn.unet, '_with_tap_plan', make)
    monkeypatch.setattr(base, '_run', spy)
    got = net(octree, pts, data)
    assert torch.equal(got, want)
    assert torch.equal(net(octree, None, data), want_nodes)
  layers = [(m.depth, n, on) for m, n, on in seen if type(m) is ocnn.OctreeConv and m.kernel_size == [3, 3, 3]]
  assert len(layers) == 2 * 47               # (conv1, and two layers of each of 15 + 8 residual blocks)
  for depth, n, on in layers:
    assert n == rows[depth] and on == (depth in planned)
  assert not hasattr(octree, 'tap_plan')
  assert int(ocnn.tc_status(octree.device).item()) == 0


def test_no_plan_that_no_layer_takes(ocnn, scene):
  """Plans serve node-major 16-bit data: for other data none is made."""
  octree, data = scene[0], node_data(scene[0], ocnn, torch.bfloat16)
  view = lambda x: ocnn.unet._with_tap_plan(octree, range(5, 10), x)
  assert view(data).tap_plan.serves(octree, 9, data.shape[2])
  for other in (data.contiguous(), data.float(), data.cpu()):
    assert view(other) is octree


def test_plans_end_with_the_pass(ocnn, scene):
  octree, _, _, pts = scene
  net, data = make_unet(ocnn, 6), node_data(octree, ocnn, torch.bfloat16)
  with torch.no_grad():
    net(octree, pts, data)                   # (weights packed, tables of the octree made)
    before = torch.cuda.memory_allocated()
    scores = net(octree, pts, data)
    size = scores.untyped_storage().nbytes()
    assert torch.cuda.memory_allocated() - before <= (size + 511) // 512 * 512


def test_a_graph_of_the_whole_pass(ocnn, scene):
  """Plans made under capture belong to the graph: a replay on other data makes them anew."""
  octree, _, _, pts = scene
  net, data = make_unet(ocnn, 7), node_data(octree, ocnn, torch.bfloat16)
  other = torch.randn_like(data)
  with torch.no_grad():
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
      want = [net(octree, pts, x) for x in (data, other)]
    torch.cuda.current_stream().wait_stream(side)
    x = data.clone(memory_format=torch.preserve_format)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
      scores = net(octree, pts, x)
    junk = torch.full((1 << 26,), 255, dtype=torch.uint8, device='cuda')     # (memory between the replays)
    for source, expected in zip((data, other, data), (want[0], want[1], want[0])):
      x.copy_(source)
      junk.fill_(255)
      graph.replay()
      assert torch.equal(scores, expected)
  torch.cuda.synchronize()
  del graph
