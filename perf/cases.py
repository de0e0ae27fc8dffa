"""What is timed: the work a user of this package has it do, through its public calls.

Every case is a dict of plain values; `kind` says which part of the package it drives:

  conv      one OctreeConv module on node data (optionally with its backward pass)
  loader    host point clouds -> normalise / transform / clip -> octrees -> merged batch
  build     point clouds on the GPU -> merged batch octree, in one call
  merge     separate octrees -> merged batch octree
  classify  point clouds on the GPU -> octree -> recorded bf16 ResNet -> logits
  resnet    host point clouds -> octree -> `ocnn.ResNet` modules (16-bit, eval) -> logits
  lenet     octree -> LeNet-style classifier in fp32 (the reference's layout) -> logits
  train     octree -> `ocnn.ResNet` in training mode, forward + cross entropy + backward (fp32)
  unet      scene octree -> `ocnn.UNet` (16-bit, non-empty nodes) -> a label row per query point

Sizes follow the package's own benchmark configurations (batches of 32 shapes with 10k-20k points at
depth 5-6, 64 clouds of 100k points at depth 8, indoor scenes of 200k points at depth 9) and the
smaller ones its tests use.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), 'o-cnn_b200'))

import ocnn  # noqa: E402
from ocnn_harness import models  # noqa: E402

FULL = 2                                  # levels 0..2 hold every node, as everywhere in the package
# node_dis, node_feature, split_label, adaptive, adp_depth, th_normal, th_distance, extrapolate,
# save_pts, key2xyz of points2octree: the defaults
BUILD = (False, False, False, False, 4, 0.1, 2.0, False, False, False)
DTYPES = {'f32': torch.float32, 'bf16': torch.bfloat16, 'f16': torch.float16}


def listed():
  return [
      # one layer on one shape: the benchmark's first configuration, and the smallest call
      dict(name='conv_f32_1x10k_d5', kind='conv', batch=1, points=10000, depth=5, cin=3, cout=32,
           dtype='f32', grad=False),
      # a training layer in fp32: forward, data gradient and weight gradient
      dict(name='conv_grad_f32_8x20k_d6', kind='conv', batch=8, points=20000, depth=6, cin=32,
           cout=64, dtype='f32', grad=True),
      # the convolution where it is a contraction: 16-bit data on a batch's finest level
      dict(name='conv_bf16_32x20k_d6', kind='conv', batch=32, points=20000, depth=6, cin=128,
           cout=128, dtype='bf16', grad=False),
      # a data loader's batch, one small ragged cloud at a time
      dict(name='loader_8x5k_d5', kind='loader', batch=8, points=5000, depth=5),
      # one scene with normals and colours
      dict(name='build_1x200k_d9', kind='build', batch=1, points=200000, depth=9, scene=True),
      # the benchmark's dense builder configuration
      dict(name='build_64x100k_d8', kind='build', batch=64, points=100000, depth=8, scene=False),
      # octrees read from a dataset, collated
      dict(name='merge_32x20k_d6', kind='merge', batch=32, points=20000, depth=6),
      # the benchmark's headline step
      dict(name='classify_bf16_32x20k_d6', kind='classify', batch=32, points=20000, depth=6),
      # serving one shape: latency of the whole chain
      dict(name='resnet_bf16_1x5k_d5', kind='resnet', batch=1, points=5000, depth=5, blocks=2,
           dtype='bf16'),
      # the benchmark's fp32 configuration
      dict(name='lenet_f32_32x10k_d5', kind='lenet', batch=32, points=10000, depth=5),
      # a training step of the classification network
      dict(name='train_f32_16x10k_d5', kind='train', batch=16, points=10000, depth=5),
      # scene segmentation
      dict(name='unet_bf16_1x200k_d9', kind='unet', batch=1, points=200000, depth=9, dtype='bf16'),
  ]


def _log(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  kind = rng.choice(['conv', 'conv', 'loader', 'build', 'merge', 'classify', 'resnet', 'lenet',
                     'train', 'unet'])
  if kind == 'conv':
    dtype = rng.choice(['f32', 'f32', 'bf16', 'f16'])
    grad = dtype == 'f32' and rng.random() < 0.5
    if dtype == 'f32':
      cin, cout = _log(rng, 3, 45), _log(rng, 8, 45)
    else:                                  # 16-bit activations come in multiples of eight channels
      cin, cout = 8 * _log(rng, 1, 22), 8 * _log(rng, 1, 22)
    return dict(kind=kind, batch=_log(rng, 1, 8 if dtype == 'f32' else 32),
                points=_log(rng, 2000, 20000), depth=rng.choice([4, 5, 6]), cin=cin, cout=cout,
                dtype=dtype, grad=grad)
  if kind == 'loader':
    return dict(kind=kind, batch=_log(rng, 1, 32), points=_log(rng, 1000, 20000),
                depth=rng.choice([5, 6]))
  if kind == 'build':
    scene = rng.random() < 0.3
    if scene:
      return dict(kind=kind, batch=rng.randint(1, 4), points=_log(rng, 20000, 200000),
                  depth=rng.choice([8, 9]), scene=True)
    return dict(kind=kind, batch=_log(rng, 1, 64), points=_log(rng, 2000, 100000),
                depth=rng.choice([5, 6, 7, 8]), scene=False)
  if kind == 'merge':
    return dict(kind=kind, batch=_log(rng, 2, 64), points=_log(rng, 2000, 40000),
                depth=rng.choice([5, 6, 7]))
  if kind == 'classify':
    return dict(kind=kind, batch=_log(rng, 1, 48), points=_log(rng, 2000, 20000),
                depth=rng.choice([5, 6]))
  if kind == 'resnet':
    return dict(kind=kind, batch=_log(rng, 1, 32), points=_log(rng, 2000, 20000),
                depth=rng.choice([5, 6]), blocks=rng.choice([1, 2, 3]),
                dtype=rng.choice(['bf16', 'f16']))
  if kind == 'lenet':
    return dict(kind=kind, batch=_log(rng, 1, 32), points=_log(rng, 1000, 10000), depth=5)
  if kind == 'train':
    return dict(kind=kind, batch=_log(rng, 2, 16), points=_log(rng, 1000, 10000),
                depth=rng.choice([4, 5]))
  return dict(kind=kind, batch=1, points=_log(rng, 20000, 200000), depth=rng.choice([7, 8, 9]),
              dtype=rng.choice(['bf16', 'f16']))


# ---- inputs ---------------------------------------------------------------------------------------
def _parts(rng, scene):
  """The solids a cloud is sampled from: kind (0 sphere, 1 box, 2 cylinder), half extents, rotation,
  offset, share of the points, colour."""
  if scene:
    n = int(rng.integers(20, 41))
    half = rng.uniform(0.03, 0.15, size=(n, 3))
    off = np.stack([rng.uniform(-0.85, 0.85, n), rng.uniform(-0.85, 0.85, n), half[:, 2] - 0.3], 1)
    half = np.concatenate([[[0.98, 0.98, 0.3]], half])
    off = np.concatenate([[[0.0, 0.0, 0.0]], off])
    kind, rot = np.ones(n + 1, np.int64), np.tile(np.eye(3), (n + 1, 1, 1))
    area = half[:, 0] * half[:, 1] + half[:, 1] * half[:, 2] + half[:, 0] * half[:, 2]
    share = area / area.sum()
  else:
    n = int(rng.integers(1, 5))
    size = rng.uniform(0.2, 0.5, size=(n, 1))
    half = size * rng.uniform(0.5, 1.0, size=(n, 3))
    kind = rng.integers(0, 3, size=n)
    rot = np.stack([np.linalg.qr(rng.normal(size=(3, 3)))[0] for _ in range(n)])
    off = rng.uniform(-0.3, 0.3, size=(n, 3))
    share = rng.dirichlet(np.full(n, 4.0))
  return kind, half, rot, off, share, rng.uniform(0.1, 0.9, size=(len(kind), 3))


def _cloud(points, seed, scene):
  """Surface points with unit normals (and colours), on the GPU, every coordinate inside (-1, 1)."""
  rng = np.random.default_rng(seed)
  gen = torch.Generator('cuda').manual_seed(seed)
  kind, half, rot, off, share, colour = (torch.as_tensor(v).cuda() for v in _parts(rng, scene))
  half, rot, off, colour = half.float(), rot.float(), off.float(), colour.float()
  part = torch.multinomial(share.float(), points, replacement=True, generator=gen)
  h = half[part]
  u = torch.rand(points, 5, device='cuda', generator=gen)
  # box: a face by its area, then a point on it
  area = torch.stack([h[:, 1] * h[:, 2], h[:, 0] * h[:, 2], h[:, 0] * h[:, 1]], 1)
  pick = u[:, 3] * area.sum(1)
  axis = (pick > area[:, 0]).long() + (pick > area[:, 0] + area[:, 1]).long()
  face = torch.nn.functional.one_hot(axis, 3).float() * torch.where(u[:, 4:] < 0.5, -1.0, 1.0)
  box = torch.where(face != 0, face, 2 * u[:, :3] - 1) * h
  # sphere
  ball = torch.nn.functional.normalize(torch.randn(points, 3, device='cuda', generator=gen), dim=1)
  # cylinder: side or caps by area
  turn = 2 * math.pi * u[:, 0]
  ring = torch.stack([turn.cos(), turn.sin(), torch.zeros_like(turn)], 1)
  up = torch.zeros_like(ring)
  up[:, 2] = torch.where(u[:, 4] < 0.5, -1.0, 1.0)
  side = (u[:, 3] * (2 * h[:, 2] + h[:, 0]) < 2 * h[:, 2])[:, None]
  tube = torch.where(side, ring * h[:, :1] + up * h[:, 2:] * (2 * u[:, 1:2] - 1),
                     ring * h[:, :1] * u[:, 1:2].sqrt() + up * h[:, 2:])
  k = kind[part][:, None]
  p = torch.where(k == 0, ball * h[:, :1], torch.where(k == 1, box, tube))
  q = torch.where(k == 0, ball, torch.where(k == 1, face, torch.where(side, ring, up)))
  r = rot[part]
  p = torch.einsum('nij,nj->ni', r, p) + off[part]
  q = torch.einsum('nij,nj->ni', r, q)
  if scene:
    p = (p + 0.002 * torch.randn(points, 3, device='cuda', generator=gen)).clamp(-0.999, 0.999)
    rgb = colour[part] + 0.03 * torch.randn(points, 3, device='cuda', generator=gen)
    return p, q, rgb.clamp(0, 1)
  p = p - 0.5 * (p.amax(0) + p.amin(0))
  return p * (0.999 / p.abs().max()), q, torch.zeros(0)


def _placed(p, q, rng):
  """One of the 48 ways a cube maps onto itself, and the points in another order: another cloud with
  another octree, of as many nodes at every level (coordinates lie on a grid that no cell boundary
  of any depth meets, so a mirrored cloud fills exactly the mirrored cells)."""
  perm = torch.as_tensor(rng.permutation(3)).cuda()
  sign = torch.as_tensor(rng.choice([-1.0, 1.0], size=3)).float().cuda()
  return p[:, perm] * sign, q[:, perm] * sign


def _clouds(case, seed, scene=False, ragged=True, place=True):
  """A batch's clouds as (xyz, normals, colours). The b-th shape and its size are always the same;
  where it stands, how it is turned or mirrored and the order of its points come from the seed."""
  rng = np.random.default_rng(seed)
  gen = torch.Generator('cuda').manual_seed(seed)
  out = []
  for b in rng.permutation(case['batch']):
    few = 0.5 + 0.5 * np.random.default_rng(int(b)).uniform() if ragged else 1.0
    p, q, c = _cloud(max(200, int(case['points'] * few)), int(b), scene)
    order = torch.randperm(p.shape[0], device='cuda', generator=gen)
    p = ((p[order] * 65536).floor() + 0.5) / 65536
    q = q[order] + 0.02 * torch.randn(q.shape, device='cuda', generator=gen)
    q = torch.nn.functional.normalize(q, dim=1)
    out.append((*(_placed(p, q, rng) if place else (p, q)), c[order] if scene else c))
  return out


def _buffers(clouds):
  """The package's host point buffers."""
  return [ocnn.points_new(p, q, c, torch.zeros(0)) for p, q, c in clouds]


def _packed(bufs):
  """The batch as points2octree_packed takes it: the clouds in one GPU buffer, where each lies, and
  their headers on the host."""
  packed, meta = ocnn.points_pack(bufs)
  return packed.cuda(), meta, torch.cat([b[:88] for b in bufs]).contiguous()


def _build(src, depth):
  return ocnn.points2octree_packed(*src, depth, FULL, *BUILD, True)


def _octree(case, seed, **kw):
  return _build(_packed(_buffers(_clouds(case, seed, **kw))), case['depth'])


def _trained(model, seed):
  """BatchNorm statistics as a trained network has them: none of them the identity."""
  gen = torch.Generator().manual_seed(seed)
  rand = lambda t, lo, hi: t.copy_(lo + (hi - lo) * torch.rand(t.shape, generator=gen))
  with torch.no_grad():
    for m in model.modules():
      if isinstance(m, (torch.nn.BatchNorm1d, torch.nn.BatchNorm2d)):
        rand(m.weight, 0.5, 1.5), rand(m.bias, -0.2, 0.2)
        rand(m.running_mean, -0.2, 0.2), rand(m.running_var, 0.5, 1.5)
  return model


def prepare(case, seed):
  ocnn.set_key_bits(64)
  torch.manual_seed(seed)
  kind, depth = case['kind'], case['depth']
  if kind == 'conv':
    octree = _octree(case, seed)
    height = int(ocnn.octree_property(octree, 'node_num', depth))
    data = torch.randn(1, case['cin'], height, 1, device='cuda')
    layer = ocnn.OctreeConv(depth, case['cin'], case['cout']).cuda()
    if case['dtype'] == 'f32':             # the reference's layout
      data.requires_grad_(case['grad'])
      grad = torch.randn(1, case['cout'], height, 1, device='cuda') if case['grad'] else None
      return dict(case=case, octree=octree, data=data, layer=layer, grad=grad)
    data = data.to(DTYPES[case['dtype']]).contiguous(memory_format=torch.channels_last)
    return dict(case=case, octree=octree, data=data, layer=layer.eval(), grad=None)
  if kind == 'loader':
    # scanned clouds: not yet centred or scaled to the unit cube
    scans = [(2.5 * p + 1.25, q, c) for p, q, c in _clouds(case, seed, place=False)]
    flags = dict(depth=depth, full_depth=FULL, distort=False)
    return dict(case=case, bufs=_buffers(scans), transform=ocnn.TransformCompose(flags))
  if kind == 'build':
    return dict(case=case, src=_packed(_buffers(_clouds(case, seed, case['scene'], False))))
  if kind == 'merge':
    make = ocnn.Points2Octree(depth, FULL)
    return dict(case=case, octrees=[make(b) for b in _buffers(_clouds(case, seed))])
  if kind == 'classify':
    net = models.GpuNet(models.resnet_params(depth, 3, 40, 2, seed=seed), 'bf16')
    return dict(case=case, src=_packed(_buffers(_clouds(case, seed, ragged=False))), net=net)
  if kind == 'resnet':
    net = _trained(ocnn.ResNet(depth, 8, 40, case['blocks']), seed).cuda().eval()
    return dict(case=case, bufs=_buffers(_clouds(case, seed)), net=net,
                make=ocnn.Points2Octree(depth, FULL))
  if kind == 'lenet':
    net = models.GpuNet(models.lenet_params(depth, 3, 40, seed=seed), 'fp32')
    return dict(case=case, octree=_octree(case, seed, ragged=False), net=net)
  if kind == 'train':
    net = _trained(ocnn.ResNet(depth, 3, 40, 1), seed).cuda().train()
    label = torch.randint(40, (case['batch'],), device='cuda')
    return dict(case=case, octree=_octree(case, seed), net=net, label=label)
  scene = _clouds(case, seed, True, False)
  octree = _build(_packed(_buffers(scene)), depth)
  net = _trained(ocnn.UNet(depth, 8, 20, nempty=True), seed).cuda().eval()
  pts = torch.cat([scene[0][0], torch.zeros(case['points'], 1, device='cuda')], 1)
  return dict(case=case, octree=octree, net=net, pts=pts)


def run(s):
  case = s['case']
  kind, depth = case['kind'], case['depth']
  if kind == 'conv':
    if s['grad'] is None:
      with torch.no_grad():
        return s['layer'](s['data'], s['octree'])
    y = s['layer'](s['data'], s['octree'])
    gx, gw = torch.autograd.grad(y, [s['data'], s['layer'].weights], s['grad'])
    return y.detach(), gx, gw
  if kind == 'loader':
    return ocnn.collate_octrees([{'octree': s['transform'](b)['octree']} for b in s['bufs']])['octree']
  if kind == 'build':
    return _build(s['src'], depth)
  if kind == 'merge':
    return ocnn.octree_batch(s['octrees'])
  if kind == 'classify':
    octree = _build(s['src'], depth)
    return octree, s['net'].forward(octree)
  if kind == 'resnet':
    with torch.no_grad():
      octree = s['make'].batch(s['bufs'])
      half = case['dtype'] == 'f16'
      data = ocnn.nn.feature_node_major(octree, 8, not half, half)
      return octree, s['net'](octree, data)
  if kind == 'lenet':
    return s['net'].forward(s['octree'])
  if kind == 'train':
    net = s['net']
    net.zero_grad(set_to_none=True)
    logits = net(s['octree'])
    loss = torch.nn.functional.cross_entropy(logits, s['label'])
    loss.backward()
    stats = [b for n, b in net.named_buffers() if 'running' in n]
    return [loss.detach()] + [p.grad for p in net.parameters()] + stats
  with torch.no_grad():
    half = case['dtype'] == 'f16'
    data = ocnn.nn.feature_node_major(s['octree'], 8, not half, half)
    return s['net'](s['octree'], s['pts'], ocnn.octree_depad(data, s['octree'], depth))


# ---- what a pass cannot do without ------------------------------------------------------------------
def _nodes(case):
  """Expected nodes per level of the batch octree: a level's occupied cells are about
  3.5 * 4^depth per shape (measured on these clouds) as far as the points reach."""
  n, batch, depth = case['points'], case['batch'], case['depth']
  if case['kind'] in ('conv', 'loader', 'merge', 'resnet', 'train'):
    n = 0.75 * n                           # ragged batches
  occupied = [3.5 * 4 ** d * (1 - math.exp(-n / (3.5 * 4 ** d))) for d in range(depth + 1)]
  return [batch * (8 ** d if d <= FULL else 8 * occupied[d - 1]) for d in range(depth + 1)], \
      [batch * o for o in occupied]


def _octree_bytes(nodes, channels, neigh=True):
  return sum(nodes) * (12 + (32 if neigh else 0)) + 4 * channels * nodes[-1]


def _resnet_flops(nodes, depth, cin, blocks, last):
  width = lambda d: 2 ** max(11 - d, 2)
  total, c = 2 * 27 * cin * width(depth) * nodes[depth], width(depth)
  for d in range(depth, last - 1, -1):
    for _ in range(blocks):
      w, b = width(d), width(d) // 4
      total += 2 * nodes[d] * (c * b + 27 * b * b + b * w + (c * w if c != w else 0))
      c = w
  return total


def _unet_flops(occ, depth):
  enc, dec = [32, 32, 64, 128, 256], [256, 256, 128, 96, 96]
  block = lambda a, b: 27 * (a * b + b * b) + (a * b if a != b else 0)
  total = 27 * 8 * 32 * occ[depth]
  for i, n in enumerate([2, 3, 4, 6]):
    h = occ[depth - i - 1]
    total += 8 * enc[i] * enc[i + 1] * h + n * block(enc[i + 1], enc[i + 1]) * h
  for i in range(4):
    h = occ[depth - 3 + i]
    total += 8 * dec[i] * dec[i + 1] * occ[depth - 4 + i]
    total += (block(dec[i + 1] + enc[-i - 2], dec[i + 1]) + block(dec[i + 1], dec[i + 1])) * h
  return 2 * total


def work(case):
  kind, depth, batch = case['kind'], case['depth'], case['batch']
  nodes, occ = _nodes(case)
  h = nodes[-1]
  cloud = batch * case['points'] * 24
  octree = _octree_bytes(nodes, 3)
  if kind == 'conv':
    size, cin, cout = (4 if case['dtype'] == 'f32' else 2), case['cin'], case['cout']
    both = 2 if case['grad'] else 1
    return {'bytes': both * (size * h * (cin + cout) + 4 * 27 * cin * cout) + 32 * h,
            'flops': (3 if case['grad'] else 1) * 2 * 27 * cin * cout * h}
  if kind == 'loader':
    return {'bytes': 0.75 * cloud + octree, 'flops': 0}
  if kind == 'build':
    if case['scene']:
      cloud, octree = cloud * 1.5, _octree_bytes(nodes, 6)
    return {'bytes': cloud + octree, 'flops': 0}
  if kind == 'merge':
    return {'bytes': octree + _octree_bytes(nodes, 3, False), 'flops': 0}
  if kind == 'classify':
    return {'bytes': cloud + octree, 'flops': _resnet_flops(nodes, depth, 3, 2, 2)}
  if kind == 'resnet':
    return {'bytes': 0.75 * cloud + octree,
            'flops': _resnet_flops(nodes, depth, 8, case['blocks'], 3)}
  if kind == 'lenet':
    chan = [3, 32, 64, 128, 256]
    flops = sum(2 * 27 * chan[i] * chan[i + 1] * nodes[depth - i] for i in range(4))
    return {'bytes': octree + 4 * 27 * sum(a * b for a, b in zip(chan, chan[1:])), 'flops': flops}
  if kind == 'train':
    return {'bytes': octree, 'flops': 3 * _resnet_flops(nodes, depth, 3, 1, 3)}
  return {'bytes': _octree_bytes(nodes, 6) + case['points'] * (16 + 40),
          'flops': _unet_flops(occ, depth)}


def tolerance(case):
  """Octrees are compared as bytes. Node data: what the data types give."""
  kind, dtype = case['kind'], case.get('dtype')
  if kind in ('loader', 'build', 'merge'):
    return 'exact'
  if kind == 'conv':
    return {'rel': {'f32': 1e-5, 'f16': 2e-3, 'bf16': 1e-2}[dtype]}
  if kind == 'lenet':
    return {'rel': 1e-5}
  if kind == 'train':
    # fp32 throughout, but sums over all nodes in an order of their own, and maxima and ReLUs whose
    # ties fall either way
    return {'rel': 1e-4}
  return {'rel': 1e-2 if dtype == 'f16' else 2e-2}
