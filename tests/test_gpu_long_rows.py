"""Long rows of a dynamic block set in the one-kernel MAS-PCG loop, where the
pairs (and with them the rows that are split over warps) change while their
number stays: the row plan is followed as it stands at each launch, through
the solver and through a handle whose caller rewrites the plan in its own
buffers, and a pattern is never taken for an earlier one.  Each solution's true
relative residual over both sets is taken in FP64 on the host; the bound is the
solve's own (a tenth more covers the drift of the recursive residual)."""

import ctypes

import numpy as np
import pytest
from scipy.sparse import coo_matrix

from yasps_b200 import _lib as L

pytestmark = pytest.mark.gpu

COUNT = 150  # pairs of a hub or a path: 151 variables, 301 blocks either way


def residual(H, x):
  A = None
  for bs in H.block_sets:
    n = bs.pattern.num_unique
    pos = bs.pattern.positions[:2 * n].cpu().numpy().astype(np.int64).reshape(-1, 2)
    val = bs.values[:9 * n].cpu().numpy().reshape(-1, 3, 3)
    r = pos[:, 0, None, None] + np.arange(3)[None, :, None] + np.zeros((1, 1, 3), dtype=np.int64)
    c = pos[:, 1, None, None] + np.arange(3)[None, None, :] + np.zeros((1, 3, 1), dtype=np.int64)
    off = pos[:, 0] != pos[:, 1]
    m = coo_matrix((np.concatenate([val.ravel(), val[off].ravel()]),
                    (np.concatenate([r.ravel(), c[off].ravel()]), np.concatenate([c.ravel(), r[off].ravel()]))),
                   shape=(H.rows, H.rows)).tocsr()
    A = m if A is None else A + m
  g = H.gradient.value.cpu().numpy()
  return np.linalg.norm(g - A @ x) / np.linalg.norm(g)


class Scene:
  """A side x side sheet (membrane, inertia) with dynamic point-point pairs among its vertices."""

  def __init__(self, side, mixed=False):
    from yasps_b200 import energies as E
    from yasps_b200.scene import scene as make_scene
    rng = np.random.default_rng(side)
    i, k = (g.ravel() for g in np.meshgrid(np.arange(side), np.arange(side), indexing="ij"))
    rest = 0.05 * np.stack([i, 0.0 * i, k], axis=1)
    x = rest + rng.uniform(-5e-3, 5e-3, rest.shape)
    self.n = len(x)
    a = (i * side + k).reshape(side, side)[:-1, :-1].ravel()
    tris = np.concatenate([np.stack([a, a + side + 1, a + side], 1), np.stack([a, a + 1, a + side + 1], 1)])
    self.sc = make_scene("long_rows")
    mesh = self.sc.addMesh("sheet")
    verts = mesh.addPrimitive("v", numInstances=self.n)
    pos = verts.addAttribute("position", rows=3, cols=1)
    pos.updateValue(x)
    consts = {}
    for name, value in (("rest", rest), ("old", rest)):
      consts[name] = verts.addConstant(name, rows=3, cols=1)
      consts[name].updateValue(value)
    mass = verts.addConstant("mass")
    mass.updateValue(np.full(self.n, 0.05))
    tri = mesh.addPrimitive("t", numInstances=len(tris))
    tc = tri.addConnectivity("c", verts, tris.astype(np.uint32), 3)
    mem = tri.addAttribute("membrane", computed_attribute=E.stvk_membrane(
        tri.addAttribute("rest", through=tc, source=consts["rest"]), tri.addAttribute("x", through=tc, source=pos),
        4e3, 4e3, 1e-3, 0.01))
    self.pairs = mesh.addPrimitive("pairs", numInstances=1, isDynamic=True)
    self.conn = self.pairs.addConnectivity("c", verts, np.array([[0, 1]], dtype=np.uint32), 2)
    dhat = 4.0 * (0.05 * side) ** 2  # beyond every pair's squared distance
    bar = self.pairs.addAttribute("barrier", computed_attribute=E.point_point(
        self.pairs.addAttribute("x", through=self.conn, source=pos), dhat, 4e-4 / dhat ** 2))
    kin = verts.addAttribute("inertia", computed_attribute=E.inertia(consts["old"], None, 0.01, pos, mass,
                                                                        gravity=(0.0, -9.8, 0.0)))
    self.sc.addEnergy(mem, projection_method=1)
    self.sc.addEnergy(bar, projection_method=1, dynamic_instances=True)
    self.sc.addEnergy(kin, projection_method=-1)
    self.sc.addMinimizeTarget([pos])
    self.sc.minimizer.setSolver("mas", mixed_spmv=mixed, stop_rule="residual")
    self.solver = self.sc.minimizer.linearSolver

  def compute(self, pairs):
    self.pairs.updateNumInstances(len(pairs))
    self.conn.updateConnectivity(np.asarray(pairs, dtype=np.uint32))
    return self.sc.minimizer.computeNumericValue()

  def solve(self, H):
    code = self.solver.computeSolution(H, H.gradient, None, tolerance=1e-6, maxIterations=5000,
                                       zero_initial_guess=True)
    assert code == 0 and self.solver.statistics["converged"]
    return self.solver.solution

  def hub(self, centre):
    other = (centre + 1 + np.arange(COUNT)) % self.n
    return np.stack([np.full(COUNT, centre), other], axis=1)

  def path(self):
    return np.stack([np.arange(COUNT), np.arange(COUNT) + 1], axis=1)


def dynamic_plan(H):
  return H.spmv_plan(H.block_sets[1])


@pytest.mark.parametrize("side", [14, 72])  # a domain a CTA and more domains than CTAs
def test_plan_rewritten_in_place(side):
  s = Scene(side)
  H = s.compute(s.path())
  assert residual(H, s.solve(H).cpu().numpy()) <= 1.1e-6
  handle, kept, values = s.solver.implementation._cache.handle, dynamic_plan(H), H.block_sets[1].values.data_ptr()
  gradient = H.gradient.value.data_ptr()
  for pairs, longest in ((s.hub(3), 151), (s.hub(s.n - 40), 151), (s.path(), 3), (s.hub(7), 151)):
    H = s.compute(pairs)
    assert H.block_sets[1].values.data_ptr() == values and H.gradient.value.data_ptr() == gradient
    new = dynamic_plan(H)
    assert int(new[0][:s.n + 1].diff().max()) == longest
    for a, b in zip(kept, new):
      assert a.numel() == b.numel()
      a.copy_(b)
    L.call("ys_pcg_set_params", handle, 1e-6, 5000)
    res = L.PcgResult()
    L.call("ys_pcg_run", handle, L.stream_ptr(), ctypes.byref(res))
    assert res.status > 0
    assert residual(H, s.solver.solution.cpu().numpy()) <= 1.1e-6


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("side", [14, 72])
def test_computes_between_solves(side, mixed):
  """Patterns whose objects and buffers are used again by later ones."""
  s = Scene(side, mixed)
  impl = s.solver.implementation
  for k in range(6):
    H = s.compute(s.path() if k % 3 == 2 else s.hub(5 + 7 * k))
    assert residual(H, s.solve(H).cpu().numpy()) <= 1.1e-6
    first, handle, pcg = id(H.block_sets[1].pattern), impl._mas.value, impl._cache.key
    for j in range(12):  # until the object's address comes round again
      H = s.compute(s.hub(60 + 5 * j + k))
      if id(H.block_sets[1].pattern) == first:
        break
    assert residual(H, s.solve(H).cpu().numpy()) <= 1.1e-6
    assert impl._cache.key != pcg


def test_more_segments_than_room():
  """Every vertex paired with every other: 400 rows of 400 entries are 1600
  segments of 128, more than the table holds (nv / 4 + 1024), so the rows are
  split in longer ones."""
  s = Scene(20)
  i, j = np.triu_indices(s.n, 1)
  H = s.compute(np.stack([i, j], axis=1))
  x = s.solve(H).clone()
  assert residual(H, x.cpu().numpy()) <= 1.1e-6
  assert bool((s.solve(H) == x).all())  # fixed order of every sum
