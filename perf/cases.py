"""Performance cases: the work a user of this library has it do, through its
public entry points.

  listed()               the cases timed by name
  draw(rng)              one more case of the same ranges
  prepare(case, seed)    the inputs and the layer a program has in hand before the call
  run(state)             one pass, and everything it computes
  work(case)             the bytes and flops one pass cannot do without
  tolerance(case)        how far another correct implementation may be off

Every pass starts from raw points, as a training step or a request does: a cloud's
bounding box, grid and neighbor lists belong to the pass, weights and upstream
gradients to the state.  All data is float32 (integers int32), the only types the
library takes.
"""
import math

import numpy as np
import torch

from tensorflow_graphics_point_clouds_b200 import classifier, custom_ops, mcconv, pc, synthetic

DEVICE = "cuda"
BANDWIDTH = 0.2


# ---- the cases -------------------------------------------------------------------

def listed():
  return [
      # The layer the library is built around: one training step of a wide
      # Monte-Carlo convolution on a full batch (the default workload of bench.py).
      dict(name="mcconv_train_wide", kind="mcconv", clouds=32, points=16384, ragged=False,
           neighbors=34.0, cin=128, mlps=1, hidden="16", cout=256, act="leaky_relu", pooled=False,
           train=True, point_grads=False),
      # The same step on a toy batch (4 x 1024 points, 8 -> 16 features): what unit
      # tests, notebooks and latency-bound callers run.
      dict(name="mcconv_train_small", kind="mcconv", clouds=4, points=1024, ragged=False,
           neighbors=5.0, cin=8, mlps=1, hidden="16", cout=16, act="leaky_relu", pooled=False,
           train=True, point_grads=False),
      # An encoder level of a network in training: four kernel MLPs of 8 units (the
      # classifier's setting), clouds of uneven size, output at the Poisson-disk
      # subsample of the input cloud.
      dict(name="mcconv_train_pooled", kind="mcconv", clouds=12, points=5003, ragged=True,
           neighbors=30.0, cin=64, mlps=4, hidden="8", cout=128, act="elu", pooled=True,
           train=True, point_grads=False),
      # A layer with two hidden layers in its kernel MLP whose points are trained
      # too: gradients of every weight and of the coordinates, the density included.
      dict(name="mcconv_train_deep_points", kind="mcconv", clouds=6, points=3001, ragged=True,
           neighbors=24.0, cin=32, mlps=1, hidden="8,16", cout=64, act="elu", pooled=False,
           train=True, point_grads=True),
      # Neighborhood construction and density estimate on scanned surfaces (long,
      # uneven neighbor lists), as preprocessing or on its own.
      dict(name="search_surface", kind="search", shape="surface", clouds=16, points=37000,
           ragged=True, dims=3, radius=0.05, max_neighbors=0, own=True, pdf_mode=0),
      # A four-level Poisson-disk hierarchy of large scenes.
      dict(name="hierarchy_poisson", kind="hierarchy", mode="poisson", clouds=8, points=100000,
           ragged=False, radius=0.025, levels=4),
      # A three-level cell-average hierarchy of a few clouds of ordinary, uneven size.
      dict(name="hierarchy_average", kind="hierarchy", mode="average", clouds=5, points=9001,
           ragged=True, radius=0.04, levels=3),
      # Inference: the three-level classification network on a batch of 1024-point shapes.
      dict(name="classifier_forward", kind="classifier", preset="three_level", clouds=32,
           points=1024),
      # One training step of a rigid kernel-point convolution (15 kernel points).
      dict(name="kpconv_train", kind="kpconv", clouds=10, points=4093, ragged=True,
           neighbors=28.0, cin=64, basis=15, cout=64, pooled=False),
      # One training step of PointConv with its learned density transform, output at
      # the subsampled cloud.
      dict(name="pointconv_train", kind="pointconv", clouds=16, points=2048, ragged=False,
           neighbors=24.0, cin=32, basis=32, cout=64, pooled=True),
      # The rest of a residual block: max pooling onto the subsampled cloud, 1x1
      # convolution, normalisation + activation, global average pooling.
      dict(name="pool_block", kind="pool", clouds=16, points=8192, ragged=False, neighbors=24.0,
           cin=128, cout=256, mode="max"),
      # The drop-in op pair BasisProj / BasisProjGrads on a prepared neighborhood, as a
      # program that keeps its own layers calls it.
      dict(name="basis_proj_op", kind="basis_proj", clouds=8, points=8192, ragged=True,
           neighbors=32.0, cin=64, basis=32),
  ]


def _log_int(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


CHANNELS = (1, 3, 8, 16, 24, 32, 48, 64, 96, 128)


def _batch(rng, most_points, least=256, largest=16384):
  """clouds (1 to 32) and points per cloud, log-uniform, at most most_points in all."""
  points = _log_int(rng, least, largest)
  clouds = _log_int(rng, 1, 32)
  clouds = max(1, min(clouds, most_points // points))
  return dict(clouds=clouds, points=points, ragged=rng.random() < 0.5)


def draw(rng):
  kind = rng.choice(["mcconv", "mcconv", "mcconv", "search", "hierarchy", "classifier", "kpconv",
                     "pointconv", "pool", "basis_proj"])
  if kind == "classifier":
    return dict(kind=kind, preset=rng.choice(["three_level", "script"]),
                clouds=_log_int(rng, 1, 32), points=_log_int(rng, 256, 2048))
  if kind == "search":
    if rng.random() < 0.5:
      return dict(kind=kind, shape="surface", dims=3, radius=round(rng.uniform(0.03, 0.06), 4),
                  max_neighbors=rng.choice([0, 0, 32]), own=rng.random() < 0.5,
                  pdf_mode=0, **_batch(rng, 300000, 1024, 40000))
    case = _batch(rng, 524288)
    dims = rng.choice([2, 3, 3, 4])
    return dict(kind=kind, shape="uniform", dims=dims,
                radius=round(_radius(rng.uniform(6, 48), case["points"], dims), 5),
                max_neighbors=rng.choice([0, 0, 16]), own=rng.random() < 0.5,
                pdf_mode=rng.choice([0, 0, 1]), **case)
  if kind == "hierarchy":
    case = _batch(rng, 500000, 1000, 100000)
    scale = (100000.0 / case["points"]) ** (1.0 / 3.0)
    return dict(kind=kind, mode=rng.choice(["poisson", "average"]), levels=rng.choice([2, 3, 4]),
                radius=round(min(0.1, 0.02 * scale * rng.uniform(0.8, 1.3)), 4), **case)
  neighbors = round(rng.uniform(8, 40), 1)
  if kind == "mcconv":
    mlps, hidden = rng.choice([(1, "8"), (1, "16"), (1, "16"), (1, "32"), (2, "8"), (4, "8"),
                               (4, "16"), (1, "8,8"), (1, "8,16"), (2, "6,8")])
    deep = "," in hidden
    basis = mlps * int(hidden.split(",")[-1])
    cin, cout = rng.choice(CHANNELS), 8 * mlps * _log_int(rng, 1, 32 // mlps)
    most = min(524288 if not deep else 32768, int(6.0e8 / (basis * cin)),
               int(8.0e10 / (basis * cin * cout)))
    train = rng.random() < 0.75
    return dict(kind=kind, neighbors=neighbors, cin=cin, mlps=mlps, hidden=hidden, cout=cout,
                act=rng.choice(["leaky_relu", "relu", "elu"]), pooled=rng.random() < 0.5,
                train=train, point_grads=train and deep and rng.random() < 0.5,
                **_batch(rng, most))
  if kind == "kpconv":
    cin, cout, basis = rng.choice(CHANNELS), 4 * _log_int(rng, 2, 64), rng.choice([13, 15, 15, 25])
    most = min(262144, int(3.0e8 / (basis * cin)), int(4.0e10 / (basis * cin * cout)))
    return dict(kind=kind, neighbors=neighbors, cin=cin, basis=basis, cout=cout,
                pooled=rng.random() < 0.5, **_batch(rng, most))
  if kind == "pointconv":
    cin, cout, basis = rng.choice(CHANNELS), 4 * _log_int(rng, 2, 64), rng.choice([8, 16, 32])
    most = min(262144, int(3.0e8 / (basis * cin)), int(4.0e10 / (basis * cin * cout)))
    return dict(kind=kind, neighbors=neighbors, cin=cin, basis=basis, cout=cout,
                pooled=rng.random() < 0.5, **_batch(rng, most))
  if kind == "pool":
    cin = rng.choice(CHANNELS[2:])
    return dict(kind=kind, neighbors=neighbors, cin=cin, cout=8 * _log_int(rng, 1, 32),
                mode=rng.choice(["max", "avg"]), **_batch(rng, min(524288, int(6.0e7 / cin))))
  cin, basis = rng.choice(CHANNELS), rng.choice([8, 16, 32, 64])
  return dict(kind=kind, neighbors=neighbors, cin=cin, basis=basis,
              **_batch(rng, min(262144, int(2.0e8 / (basis * cin)))))


# ---- inputs -----------------------------------------------------------------------

def _sizes(case):
  """Points per cloud: all equal, or (ragged) between half and one and a half times
  the nominal number; fixed by the case, so that work() knows them."""
  n = case["points"]
  if not case.get("ragged"):
    return [n] * case["clouds"]
  r = np.random.default_rng(case["clouds"] * 1000003 + n)
  return [int(v) for v in r.integers(max(1, n // 2), n + n // 2 + 1, case["clouds"])]


def _total(case):
  return sum(_sizes(case))


def _ball(dims, radius):
  return math.pi ** (dims / 2.0) / math.gamma(dims / 2.0 + 1.0) * radius ** dims


def _radius(neighbors, points, dims=3):
  """Radius at which a point in the middle of `points` uniform ones has `neighbors`."""
  share = min(0.25, neighbors / float(points))
  return (share / _ball(dims, 1.0)) ** (1.0 / dims)


def _pairs_per_point(case, dims=3):
  """Mean list length on uniform clouds of the unit cube, edges allowed for."""
  r = case["radius"] if "radius" in case else _radius(case["neighbors"], case["points"], dims)
  inner = max(0.3, 1.0 - 0.1875 * dims * r)
  sizes = np.array(_sizes(case), dtype=np.float64)
  return float((sizes * np.maximum(1.0, sizes * _ball(dims, r) * inner)).sum() / sizes.sum())


# The number of neighbor pairs and of samples follows from the points, and two inputs
# of one case have to give arrays of the same size.  The geometry of a case is therefore
# drawn from the case alone, and the seed changes what leaves those numbers alone: the
# order of the points inside a cloud, the order of the clouds, the unit of length;
# and of course features, weights and gradients.

def _generator(seed):
  g = torch.Generator(device=DEVICE)
  g.manual_seed(int(seed))
  return g


def _geometry(case):
  return _generator(7919 * _total(case) + case["clouds"])


def _shuffled(points, ids, g):
  """The points of every cloud in another order."""
  key = ids.double() + torch.rand(ids.shape, generator=g, device=DEVICE, dtype=torch.float64)
  return points[torch.argsort(key)]


def _clouds_reordered(points, sizes, g):
  """The clouds in another order (points, batch ids)."""
  order = torch.randperm(len(sizes), generator=g, device=DEVICE).tolist()
  parts = torch.split(points, sizes)
  return torch.cat([parts[i] for i in order]), _batch_ids([sizes[i] for i in order])


def _batch_ids(sizes):
  return torch.repeat_interleave(torch.arange(len(sizes), dtype=torch.int32, device=DEVICE),
                                 torch.tensor(sizes, device=DEVICE))


def _uniform(sizes, g, dims=3):
  return torch.rand((sum(sizes), dims), generator=g, device=DEVICE), _batch_ids(sizes)


def _surfaces(sizes, g, shapes=8, noise=0.005):
  """Points on the surfaces of random spheres and boxes (centres uniform in the unit
  cube, sizes uniform in [0.1, 0.4]) plus Gaussian noise, as synthetic.surface_clouds."""
  n, b = sum(sizes), len(sizes)
  ids = _batch_ids(sizes)
  centre = torch.rand((b, shapes, 3), generator=g, device=DEVICE)
  size = 0.1 + 0.3 * torch.rand((b, shapes), generator=g, device=DEVICE)
  shape = torch.randint(0, shapes, (n,), generator=g, device=DEVICE)
  sphere = torch.randn((n, 3), generator=g, device=DEVICE)
  sphere = 0.5 * sphere / sphere.norm(dim=1, keepdim=True)
  box = torch.rand((n, 3), generator=g, device=DEVICE) - 0.5
  face = torch.randint(0, 6, (n,), generator=g, device=DEVICE)
  box.scatter_(1, (face // 2)[:, None], ((face % 2).float() - 0.5)[:, None])
  unit = torch.where((shape % 2 == 0)[:, None], sphere, box)
  pts = centre[ids.long(), shape] + size[ids.long(), shape][:, None] * unit
  return pts + noise * torch.randn((n, 3), generator=g, device=DEVICE), ids


def _mixture(sizes, g, components=12):
  """Points of anisotropic Gaussian mixtures, as synthetic.gaussian_mixture_clouds."""
  n, b = sum(sizes), len(sizes)
  ids = _batch_ids(sizes)
  centre = torch.rand((b, components, 3), generator=g, device=DEVICE)
  sigma = 0.01 + 0.09 * torch.rand((b, components, 3), generator=g, device=DEVICE)
  comp = torch.randint(0, components, (n,), generator=g, device=DEVICE)
  pts = (centre[ids.long(), comp] +
         sigma[ids.long(), comp] * torch.randn((n, 3), generator=g, device=DEVICE))
  return pts, ids


def _normal(g, *shape):
  return torch.randn(shape, generator=g, device=DEVICE)


def _glorot(g, *shape):
  lim = math.sqrt(6.0 / (shape[-2] + shape[-1]))
  return (2.0 * torch.rand(shape, generator=g, device=DEVICE) - 1.0) * lim


def _clouds(case, g):
  """Input cloud, output cloud (the input's Poisson-disk subsample where the layer
  pools) and radius of a layer."""
  sizes = _sizes(case)
  points, ids = _uniform(sizes, _geometry(case))
  radius = _radius(case["neighbors"], case["points"])
  s = dict(clouds=len(sizes), points=_shuffled(points, ids, g), batch_ids=ids, radius=radius)
  if case.get("pooled") or case["kind"] == "pool":
    coarse = pc.PointHierarchy(pc.PointCloud(points, ids, len(sizes)), [radius],
                               "poisson")._point_clouds[1]
    s["out_points"], s["out_batch_ids"] = coarse._points, coarse._batch_ids
  else:
    s["out_points"] = s["points"]
  return s


def prepare(case, seed):
  kind, g = case["kind"], _generator(seed)
  if kind == "classifier":
    preset = classifier.PRESETS[case["preset"]]
    pts, ids = synthetic.unit_sphere_shapes(case["clouds"], case["points"], seed)
    weights = synthetic.small_classifier_weights(seed, preset["feature_sizes"],
                                                 head_layers=preset["head_layers"])
    net = classifier.SmallClassifier(weights, preset["radii"], torch.device(DEVICE),
                                     preset["pool_before_head"])
    return dict(kind=kind, net=net, clouds=case["clouds"], points=torch.from_numpy(pts).to(DEVICE),
                batch_ids=torch.from_numpy(ids).to(DEVICE),
                features=torch.ones((len(pts), 1), device=DEVICE))
  if kind == "search":
    sizes = _sizes(case)
    make = _surfaces if case["shape"] == "surface" else lambda s, gen: _uniform(s, gen, case["dims"])
    fixed = _geometry(case)
    points, ids = make(sizes, fixed)
    s = dict(case, clouds=len(sizes), points=_shuffled(points, ids, g), batch_ids=ids)
    if not case["own"]:
      # queries beside the cloud: every third point, moved a little
      s["samples"] = points[::3] + 0.3 * case["radius"] * _normal(fixed, *points[::3].shape)
      s["sample_ids"] = ids[::3].contiguous()
    return s
  if kind == "hierarchy":
    # scenes some way from the origin, in units from 1 to 1/128 of the case's
    unit = 2.0 ** (seed % 8)
    points, _ = _mixture(_sizes(case), _geometry(case))
    points, ids = _clouds_reordered((points + 1.0) * unit, _sizes(case), g)
    return dict(kind=kind, clouds=case["clouds"], points=points, batch_ids=ids, mode=case["mode"],
                radii=[unit * case["radius"] * 2 ** i for i in range(case["levels"])])
  s = _clouds(case, g)
  n, ns = s["points"].shape[0], s["out_points"].shape[0]
  s["kind"], s["pooled"] = kind, bool(case.get("pooled")) or kind == "pool"
  s["features"] = _normal(g, n, case["cin"])
  cin = case["cin"]
  if kind == "mcconv":
    widths = [3] + [int(h) for h in case["hidden"].split(",")]
    mlps = case["mlps"]
    w = [_glorot(g, mlps, a, b) for a, b in zip(widths[:-1], widths[1:])]
    b = [0.1 * _normal(g, mlps, 1, h) for h in widths[1:]]
    wf = _glorot(g, mlps, cin * widths[-1], case["cout"] // mlps)
    one = len(w) == 1
    s["layer"] = mcconv.MCConv(w[0] if one else w, b[0] if one else b, wf, cin,
                               non_linearity_type=case["act"])
    s["train"], s["point_grads"] = case["train"], case["point_grads"]
    s["out_grads"] = _normal(g, ns, case["cout"]) if case["train"] else None
  elif kind == "kpconv":
    kernel_points = _normal(g, case["basis"], 3)
    kernel_points = kernel_points / kernel_points.norm(dim=1, keepdim=True).clamp(min=1.0)
    kernel_points[0] = 0.0
    s["layer"] = mcconv.KPConv(kernel_points, _glorot(g, cin * case["basis"], case["cout"]), cin)
    s["out_grads"] = _normal(g, ns, case["cout"])
  elif kind == "pointconv":
    s["layer"] = mcconv.PointConv(
        _normal(g, 3, case["basis"]), 0.1 * _normal(g, 1, case["basis"]),
        _glorot(g, cin * case["basis"], case["cout"]), [_normal(g, 1, 16), _normal(g, 16, 1).abs()],
        [_normal(g, 1, 16).abs(), torch.ones((1, 1), device=DEVICE)], cin)
    s["out_grads"] = _normal(g, ns, case["cout"])
  elif kind == "pool":
    s["mode"] = case["mode"]
    s["weights"], s["bias"] = _glorot(g, cin, case["cout"]), 0.1 * _normal(g, 1, case["cout"])
  else:
    grid = pc.Grid(pc.PointCloud(s["points"], s["batch_ids"], s["clouds"]), s["radius"])
    neigh = pc.Neighborhood(grid, s["radius"], grid._point_cloud)
    s["neighbors"], s["ranges"] = neigh._original_neigh_ids, neigh._samples_neigh_ranges
    s["basis"] = _normal(g, s["neighbors"].shape[0], case["basis"])
    s["out_grads"] = _normal(g, ns, cin, case["basis"])
  return s


# ---- one pass --------------------------------------------------------------------

def run(s):
  kind = s["kind"]
  if kind == "classifier":
    return s["net"].forward(s["points"], s["batch_ids"], s["clouds"], s["features"])
  if kind == "basis_proj":
    args = (s["basis"], s["features"], s["neighbors"], s["ranges"])
    out = custom_ops.basis_proj(*args)
    return (out,) + tuple(custom_ops.basis_proj_grads(*args, s["out_grads"]))
  cloud = pc.PointCloud(s["points"], s["batch_ids"], s["clouds"])
  if kind == "search":
    samples = None if s["own"] else pc.PointCloud(s["samples"], s["sample_ids"], s["clouds"])
    neigh = pc.grid_neighborhood(cloud, s["radius"], samples, s["max_neighbors"])
    neigh.compute_pdf(bandwidth=BANDWIDTH, mode=s["pdf_mode"])
    return dict(ranges=neigh._samples_neigh_ranges, neighbors=neigh._neighbors,
                density=neigh.point_pdf())
  if kind == "hierarchy":
    hier = pc.PointHierarchy(cloud, s["radii"], s["mode"])
    levels = hier._point_clouds[1:]
    return dict(points=[c._points for c in levels], batch_ids=[c._batch_ids for c in levels],
                indices=list(hier._sample_indices))
  out_cloud = cloud
  if s["pooled"]:
    out_cloud = pc.PointCloud(s["out_points"], s["out_batch_ids"], s["clouds"])
  if kind == "pool":
    x = mcconv.local_pool(s["features"], cloud, out_cloud, s["radius"], s["mode"])
    y = mcconv.conv1x1(x, s["weights"], s["bias"])
    y = mcconv.scale_bias_activation_(y, 0.999, None, 0.3)
    return dict(pooled=x, features=y, per_cloud=mcconv.global_pool(y, out_cloud, "avg"))
  layer = s["layer"]
  if kind != "mcconv":
    out = layer.forward(s["features"], cloud, out_cloud, s["radius"])
    return (out,) + tuple(layer.backward(s["out_grads"]))
  if not s["point_grads"]:
    out = layer.forward(s["features"], cloud, out_cloud, s["radius"], bandwidth=BANDWIDTH,
                        keep_for_backward=s["train"])
    return (out,) + tuple(layer.backward(s["out_grads"])) if s["train"] else out
  neigh = layer.build_neighborhood(cloud, out_cloud, s["radius"])
  out = layer.forward(s["features"], cloud, out_cloud, s["radius"], neighborhood=neigh,
                      bandwidth=BANDWIDTH)
  grads = layer.backward(s["out_grads"], point_grads=True)
  return (out,) + tuple(grads) + (neigh.pdf_point_grads(grads[-1], bandwidth=BANDWIDTH),)


# ---- what a pass cannot do without --------------------------------------------------

def _subsample(case):
  """Number of points a Poisson-disk subsample at the layer's radius keeps (about
  three per ball of that radius in the bulk of a uniform cloud)."""
  per_cloud = 3.0 / _ball(3, _radius(case["neighbors"], case["points"]))
  return sum(min(float(v), per_cloud) for v in _sizes(case))


def work(case):
  kind = case["kind"]
  if kind == "classifier":
    preset = classifier.PRESETS[case["preset"]]
    f, n = preset["feature_sizes"], case["clouds"] * case["points"]
    levels = len(preset["radii"])
    weights = sum(a * b * (32 if i < levels else 1) for i, (a, b) in enumerate(zip(f, f[1:])))
    weights += sum(v * v for v in f[1:levels])
    flops, rows = 0.0, float(n)
    for i in range(levels):
      rows = max(float(case["clouds"]), min(rows, case["clouds"] * 8.0 / preset["radii"][i] ** 2))
      flops += 2.0 * rows * 32 * f[i] * f[i + 1] + (2.0 * rows * f[i + 1] ** 2 if i < levels - 1 else 0)
    return {"bytes": 20.0 * n + 4.0 * weights + 4.0 * case["clouds"] * f[-1], "flops": flops}
  n = _total(case)
  if kind == "hierarchy":
    kept = [n / (4.0 ** (i + 1)) for i in range(case["levels"])]
    return {"bytes": 16.0 * n + sum(20.0 * v for v in kept), "flops": 30.0 * n}
  if kind == "search":
    d = case["dims"]
    if case["shape"] == "surface":
      # mean over a cloud of 8 patches of mean area ~0.15 each, blurred by the noise
      pairs = n * max(1.0, n / case["clouds"] * math.pi * case["radius"] ** 2 / 1.1)
    else:
      pairs = n * _pairs_per_point(case, d)
    samples = n if case["own"] else (n + 2) // 3
    listed_pairs = pairs * samples / n
    if case["max_neighbors"]:
      listed_pairs = min(listed_pairs, samples * float(case["max_neighbors"]))
    # the density of every point takes its own neighborhood whatever the samples are
    return {"bytes": n * (4.0 * d + 8.0) + samples * (0.0 if case["own"] else 4.0 * d + 4.0) +
                     4.0 * samples + 8.0 * listed_pairs,
            "flops": (3.0 * d) * (pairs + listed_pairs) + 4.0 * d * pairs}
  pairs = n * _pairs_per_point(case)
  cin, cout = case["cin"], case.get("cout", 0)
  pooled = case.get("pooled") or kind == "pool"
  ns = _subsample(case) if pooled else float(n)
  list_pairs = pairs * ns / n
  if kind == "pool":
    return {"bytes": n * (16.0 + 4.0 * cin) + ns * (16.0 + 4.0 * cin + 4.0 * cout) +
                     4.0 * cin * cout + 4.0 * case["clouds"] * cout,
            "flops": 9.0 * list_pairs + list_pairs * cin + 2.0 * ns * cin * cout}
  if kind == "basis_proj":
    k = case["basis"]
    return {"bytes": list_pairs * (8.0 + 4.0 * k + 4.0 * k) + 4.0 * ns + 8.0 * n * cin +
                     8.0 * ns * cin * k,
            "flops": 6.0 * list_pairs * cin * k}
  if kind == "mcconv":
    widths = [3] + [int(h) for h in case["hidden"].split(",")]
    k = case["mlps"] * widths[-1]
    mlp = 2.0 * case["mlps"] * sum(a * b for a, b in zip(widths, widths[1:]))
    train = case["train"]
  else:
    k = case["basis"]
    mlp, train = (10.0 if kind == "kpconv" else 6.0) * k, True
  weights = 4.0 * k * cin * cout
  forward = n * (16.0 + 4.0 * cin) + (ns * 16.0 if pooled else 0.0) + weights + 4.0 * ns * cout
  flops = list_pairs * (9.0 + mlp + 2.0 * cin * k) + 2.0 * ns * k * cin * cout
  if kind != "kpconv":
    flops += pairs * 21.0      # the density estimate over every point's own neighborhood
  if not train:
    return {"bytes": forward, "flops": flops}
  backward = 4.0 * ns * cout + 4.0 * n * cin + weights
  flops += list_pairs * (2.0 * mlp + 4.0 * cin * k) + 4.0 * ns * k * cin * cout
  if case.get("point_grads"):
    backward += 24.0 * n + 4.0 * list_pairs
    flops += pairs * 24.0
  return {"bytes": forward + backward, "flops": flops}


def tolerance(case):
  kind = case["kind"]
  if kind in ("hierarchy", "search"):
    # whole numbers the same; densities and averages are short float32 sums
    return {"rel": 2e-6, "max": 5e-5}
  # float32 sums of up to 1e7 terms and products in float32 accuracy; single values that
  # cancel, or whose activation sits within rounding of its kink, show up to the library's
  # parity bound of 1e-4 on either side
  return {"rel": 2e-5, "max": 2e-4}
