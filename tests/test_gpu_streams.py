"""Solves in flight on several streams: each takes a part of the chip, and the
solution has the bits of a solve that has the chip to itself."""

import threading

import numpy as np
import pytest

from tests import test_gpu_long_rows as long_rows
from yasps_b200 import _lib as L
from yasps_b200 import scenes

pytestmark = pytest.mark.gpu


def make(side, mixed, seed, **options):
  import torch
  stream = torch.cuda.Stream()
  with torch.cuda.stream(stream):
    sc, _ = scenes.fem_scene(scenes.fem_cube(side, noise=0.01, seed=seed))
    solver = sc.minimizer.setSolver("mas", mixed_spmv=mixed, stop_rule="residual", **options)
    x = sc.minimizeEnergy(tolerance=1e-6, maxIterations=2000)[0].clone()
  stream.synchronize()
  return stream, sc, solver, x


def make_two_sets(side, mixed):
  """A second block set with a row of several segments."""
  import torch
  stream = torch.cuda.Stream()
  with torch.cuda.stream(stream):
    s = long_rows.Scene(side, mixed)
    x = s.solve(s.compute(s.hub(11))).clone()
  stream.synchronize()
  return stream, s, s.solver, x


# one domain, a domain a CTA (tens of CTAs; the whole chip), warps over many
# domains, one level, two block sets
@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("side,form", [(3, "levels"), (9, "levels"), (16, "levels"), (25, "levels"),
                                       (17, "one level"), (25, "one level"), (14, "two sets"), (72, "two sets")])
def test_solution_does_not_depend_on_solves_in_flight(side, form, mixed):
  """Launched without waiting in between, so 1, 2, 3, 4 and 5 are in flight."""
  if form == "two sets":
    solves = [make_two_sets(side, mixed) for _ in range(5)]
  else:
    options = dict(max_levels=1, global_coarse_domain=False) if form == "one level" else {}
    solves = [make(side, mixed, 1, **options) for _ in range(5)]
  handles = [s[2].implementation._cache.handle for s in solves]
  work = [s[2].implementation for s in solves]
  before = []
  for (stream, _, _, _), h, w in zip(solves, handles, work):  # alone: status waits
    res = L.PcgResult()
    L.call("ys_pcg_launch", h, stream.cuda_stream)
    L.call("ys_pcg_status", h, stream.cuda_stream, res)
    target = w._mixed[1] if mixed else w.solution
    before.append((target, target.cpu().numpy().copy(), int(res.iterations)))
    assert np.array_equal(before[0][1], before[-1][1])
  for _ in range(3):
    for target, _, _ in before:
      target.zero_()
    import torch
    torch.cuda.synchronize()
    for (stream, _, _, _), h in zip(solves, handles):
      L.call("ys_pcg_launch", h, stream.cuda_stream)
    for (stream, _, _, _), h, (target, x, its) in zip(solves, handles, before):
      res = L.PcgResult()
      L.call("ys_pcg_status", h, stream.cuda_stream, res)
      assert res.status >= 0 and int(res.iterations) == its
      assert np.array_equal(target.cpu().numpy(), x)


def test_threads():
  solves = [make(side, mixed, side) for side in (12, 20, 25) for mixed in (True, False)]
  failed = []

  def work(stream, sc, solver, x):
    import torch
    try:
      with torch.cuda.stream(stream):
        for _ in range(10):
          y = sc.minimizeEnergy(tolerance=1e-6, maxIterations=500)[0]
          assert bool((y == x).all())
    except Exception as error:  # noqa: BLE001
      failed.append(error)

  threads = [threading.Thread(target=work, args=s) for s in solves]
  for t in threads:
    t.start()
  for t in threads:
    t.join()
  assert not failed, failed
