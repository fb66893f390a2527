"""The closed-form vertex-tuple energies one kind at a time (in a mixed scene
the stiffest kind's entries hide the others'): gradient and Hessian of a scene
that holds the kind alone against the oracle's autograd, for one element, for
one past a warp and, for the friction kinds, with every element repeating a
vertex (merged records; a repeated vertex puts the distance, the area or the
hinge's angle of the others at a singular point, where their energies have no
derivatives).  Bound 1e-12 of the kind's largest entry, the suite's bar for
FP64 element Hessians."""

from types import SimpleNamespace

import numpy as np
import pytest

from oracle import projection
from oracle import vertex_energies as ve
from tests.vertex_scene import VertexScene

pytestmark = pytest.mark.gpu


def scene_of(vs, kind, conn, params, aux, lag, method):
  from yasps_b200 import energies as E
  from yasps_b200.scene import scene as make_scene
  sc = make_scene("one_kind")
  mesh = sc.addMesh("m")
  verts = mesh.addPrimitive("v", numInstances=len(vs.x))
  pos = verts.addAttribute("position", rows=3, cols=1)
  pos.updateValue(vs.x)
  other = verts.addConstant("aux", rows=3, cols=1)
  other.updateValue(vs.rest if aux == "rest" else vs.x_old)
  prim = mesh.addPrimitive("e", numInstances=len(conn))
  c = prim.addConnectivity("c", verts, conn.astype(np.uint32), conn.shape[1])
  x = prim.addAttribute("x", through=c, source=pos)
  r = prim.addAttribute("r", through=c, source=other)
  if lag is not None:
    q = prim.addConstant("lag", rows=9, cols=1)
    q.updateValue(lag)
    make = {8: E.friction_point_triangle, 9: E.friction_point_edge, 10: E.friction_edge_edge,
            11: E.friction_point_point}[kind]
    e = make(x, r, *params, q)
  elif kind == 5:
    e = E.bending(x, r, *params)
  elif kind in (6, 7):
    e = (E.baraff_witkin if kind == 6 else E.stvk_membrane)(r, x, *params)
  else:
    e = {1: E.point_point, 2: E.point_edge, 3: E.point_triangle, 4: E.edge_edge}[kind](x, *params)
  sc.addEnergy(prim.addAttribute("energy", computed_attribute=e), projection_method=method)
  sc.addMinimizeTarget([pos])
  return sc


CASES = [(kind, count) for kind in range(1, 12) for count in (1, 33)] + [(kind, "merged") for kind in range(8, 12)]


@pytest.mark.parametrize("method", [0, 1, 2])
@pytest.mark.parametrize("kind,count", CASES)
def test_kind_alone(kind, count, method):
  vs = VertexScene(m=6, seed=11, membrane="baraff_witkin" if kind != 7 else "stvk")
  _, conn, params, aux, lag = next(t for t in vs.terms() if t[0] == kind)
  merged = count == "merged"
  n = 3 if merged else count
  take = np.arange(n) % len(conn)
  conn, lag = conn[take].copy(), None if lag is None else lag[take]
  if merged:
    conn[:, -1] = conn[:, 0]
  sc = scene_of(vs, kind, conn, params, aux, lag, method)
  H = sc.minimizer.computeNumericValue()
  src = {"rest": vs.rest, "old": vs.x_old, None: None}[aux]
  _, gl, hl = ve.energy_grad_hess(kind, vs.x[conn], None if src is None else src[conn], params, lag)
  h0 = hl
  if method:
    hl = projection.project_spd(hl, method)
  D, g = np.zeros((vs.n, vs.n)), np.zeros(vs.n)
  for t, c in enumerate(conn):
    i = (3 * np.asarray(c)[:, None] + np.arange(3)).ravel()
    np.add.at(D, (i[:, None], i[None]), hl[t])
    np.add.at(g, i, gl[t])
  pos = H.block_positions.cpu().numpy().astype(np.int64).reshape(-1, 2)
  val = H.blocks_flattened.cpu().numpy()[:9 * len(pos)].reshape(-1, 3, 3)
  dev = np.zeros_like(D)
  for (r, c), b in zip(pos, val):
    dev[r:r + 3, c:c + 3] += b
    if r != c:
      dev[c:c + 3, r:r + 3] += b.T
  assert np.abs(H.gradient.value.cpu().numpy() - g).max() <= 1e-12 * np.abs(gl).max()
  # projecting: negative eigenvalues within the PSD test's absolute tolerance
  # (1e-10, at most 3 of them in sums of 3 elements an entry) may stay
  slack = 1e-9 if method and np.abs(hl).max() < 1e-3 else 0.0
  largest = max(np.abs(h0).max(), np.abs(hl).max())  # rounding follows the unprojected entries
  assert np.abs(dev - D).max() <= len(conn) * 1e-12 * largest + slack


def random_elements(kind, n, rng):
  """Elements of the kind far from flat, straight and still ones, with vertices of their own."""
  wide = lambda *shape: rng.uniform(-0.25, 0.25, shape)
  tri = np.array([[0.0, 0.0, 0.0], [1.0, 0.0, 1.0], [1.0, 0.0, 0.0]])  # normal along +y
  shapes = {1: [[0.0, 0.9, 0.0], [0.0, 0.0, 0.0]], 2: [[0.5, 0.9, 0.5], [0.0, 0.0, 0.0], [1.0, 0.0, 1.0]],
            3: [[0.7, 0.9, 0.4], *tri], 4: [[0.0, 0.9, 0.5], [1.0, 0.9, 0.5], [0.5, 0.0, 0.0], [0.5, 0.0, 1.0]],
            5: [[0.0, 0.0, 0.0], [0.0, 0.0, 1.0], [0.9, 0.3, 0.5], [-0.9, 0.3, 0.5]], 6: tri, 7: tri}
  like = {8: 3, 9: 2, 10: 4, 11: 1}
  base = np.asarray(shapes[like.get(kind, kind)])
  A = len(base)
  x = base + wide(n, A, 3)
  rest = base + 0.2 * wide(n, A, 3)
  params = {1: (2.5, 3.0), 2: (2.5, 3.0), 3: (2.5, 3.0), 4: (2.5, 3.0), 5: (3.0, 0.1), 6: (2e3, 1e3, 0.1, 0.1),
            7: (5e3, 2e3, 0.1, 0.1)}.get(kind, (4.0, 0.1, 0.3))
  old = x + 0.4 * wide(n, A, 3)  # slides of up to about twice the stick range, 0.2
  lag = None
  if kind >= 8:
    q, _ = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    lag = np.concatenate([rng.uniform(0.1, 0.45, (n, 2)), q[:, :, 0], q[:, :, 1], rng.uniform(1.0, 2.0, (n, 1))], 1)
  return x, rest, old, params, lag


@pytest.mark.parametrize("kind", range(1, 12))
def test_blocks_of_random_elements(kind):
  """Every block of many elements that share no vertex, unprojected, each
  element against its own largest entry: 3e-12 allows some 300 roundings on
  terms a hundred times the entries they cancel to."""
  n = 1001
  x, rest, old, params, lag = random_elements(kind, n, np.random.default_rng(kind))
  A = x.shape[1]
  aux = "rest" if kind in (5, 6, 7) else "old" if kind >= 8 else None
  src = {"rest": rest, "old": old, None: None}[aux]
  vs = SimpleNamespace(x=x.reshape(-1, 3), rest=rest.reshape(-1, 3), x_old=old.reshape(-1, 3))
  sc = scene_of(vs, kind, np.arange(n * A).reshape(n, A), params, aux, lag, 0)
  H = sc.minimizer.computeNumericValue()
  _, gl, hl = ve.energy_grad_hess(kind, x, src, params, lag)
  pos = H.block_positions.cpu().numpy().astype(np.int64).reshape(-1, 2)
  val = H.blocks_flattened.cpu().numpy()[:9 * len(pos)].reshape(-1, 3, 3)
  t, a, b = pos[:, 0] // (3 * A), pos[:, 0] // 3 % A, pos[:, 1] // 3 % A
  assert len(pos) == n * A * (A + 1) // 2 and np.all(pos[:, 1] // (3 * A) == t)
  want = hl.reshape(n, A, 3, A, 3)[t, a, :, b]
  scale = np.abs(hl).max(axis=(1, 2))
  assert np.all(scale > 0)
  assert (np.abs(val - want).max(axis=(1, 2)) / scale[t]).max() <= 3e-12
  g = H.gradient.value.cpu().numpy().reshape(n, -1)
  # (a rounding of a coordinate moves the gradient by the Hessian's share of it)
  assert (np.abs(g - gl).max(axis=1) / np.maximum(np.abs(gl).max(axis=1), scale)).max() <= 3e-12
