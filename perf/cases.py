"""Timed cases: the Newton inner loop through its public entry points.

The framework serves simulation codes that take Newton steps: evaluate the
energies, assemble the projected Hessian, solve ``H x = g``.  The cases are
two whole steps at the ends of the size range, one on the mixed cloth + body +
contact scene, and the parts a program calls by themselves: ``hessian.compute``
(volumes, contacts, and contact sets that change every call), the linear
solvers, ``hessian.spmv``, the energy total of a line search, the shape
Jacobian of a differentiable simulation, and the serving form.

Sizes and materials are those of this repository's benchmark, serving streams
and tests: cube sides 8..64, cloth sides 64..256, 10k..200k contact pairs.
"""

import dataclasses
import functools
import warnings

import numpy as np
import torch

from yasps_b200 import energies as E
from yasps_b200 import scenes, serving
from yasps_b200.graph import resolve_leaf_children
from yasps_b200.hessian import vector
from yasps_b200.jacobian import differentiator
from yasps_b200.scene import scene as make_scene
from yasps_b200.solver import solver as make_solver

TOL = 1e-6          # true relative residual of the benchmark's solves
MAX_IT = 20000


def listed():
  return [
      # a whole Newton step of the smallest scenes: launches and latency
      dict(name="step_fem9", kind="step", side=9, young=1e5, poisson=0.4, noise=0.01, mixed=True),
      # the benchmark's headline step (774k DoF, 1.5M tetrahedra, FP32 + refinement)
      dict(name="step_fem64", kind="step", side=64, young=1e6, poisson=0.45, noise=0.005, mixed=True),
      # the mixed scene: cloth on an obstacle under 16 affine bodies, 200k barrier pairs
      dict(name="step_cloth256", kind="cloth_step", side=256, pairs=200_000, bodies=16, mixed=True),
      # gradient + Hessian of a volume, eigenvalues clamped, FP64 only (odd side)
      dict(name="compute_fem41", kind="compute", side=41, young=1e5, poisson=0.4, noise=0.01, method=2),
      # gradient + Hessian of cloth with a static contact set
      dict(name="compute_contact181", kind="contact", side=181, pairs=100_000, method=1),
      # the same with contact pairs that change every call: pattern rebuilt each time
      dict(name="compute_dynamic96", kind="dynamic", side=96, pairs=40_000, method=1),
      # the drop-in solver: MAS preconditioner rebuild + FP64 PCG of an assembled system
      dict(name="solve_mas33", kind="solve", side=33, young=1e6, poisson=0.45, noise=0.005, method="mas"),
      # block-Jacobi PCG, the reference's other solver
      dict(name="solve_jacobi25", kind="solve", side=25, young=1e5, poisson=0.4, noise=0.01, method="jacobian"),
      # one symmetric block product in FP64
      dict(name="spmv_fem57", kind="spmv", side=57, young=1e5, poisson=0.4, noise=0.01),
      # energy total of a line-search trial point
      dict(name="energy_fem48", kind="energy", side=48, young=1e5, poisson=0.4, noise=0.01),
      # shape derivative d2E/dx dX and its two products
      dict(name="shape_fem20", kind="shape", side=20, young=1e5, poisson=0.4, noise=0.01),
      # the serving form: 16 requests of four cube sides at once
      dict(name="serve_16", kind="serve", sides="8,14,21,28", requests=16),
  ]


def draw(rng):
  def between(lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))

  material = dict(young=round(10 ** rng.uniform(4, 6), 1), poisson=round(rng.uniform(0.3, 0.45), 3),
                  noise=rng.choice([0.005, 0.01]))
  kind = rng.choice(["step", "cloth_step", "compute", "contact", "dynamic", "solve", "spmv", "energy", "shape", "serve"])
  if kind == "step":
    return dict(kind=kind, side=between(8, 60), mixed=rng.random() < 0.7, **material)
  if kind == "cloth_step":
    return dict(kind=kind, side=between(64, 240), pairs=between(10_000, 180_000), bodies=rng.randint(0, 15),
                mixed=rng.random() < 0.7)
  if kind == "compute":
    return dict(kind=kind, side=between(8, 62), method=rng.choice([1, 2, -1]), **material)
  if kind == "contact":
    return dict(kind=kind, side=between(64, 250), pairs=between(10_000, 190_000), method=rng.choice([1, 2]))
  if kind == "dynamic":
    return dict(kind=kind, side=between(64, 180), pairs=between(2_000, 100_000), method=rng.choice([1, 2]))
  if kind == "solve":
    return dict(kind=kind, side=between(8, 45), method=rng.choice(["mas", "mas", "jacobian"]), **material)
  if kind == "shape":
    return dict(kind=kind, side=between(8, 30), **material)
  if kind == "serve":
    sides = sorted(rng.sample(range(8, 33), rng.randint(2, 4)))
    return dict(kind=kind, sides=",".join(map(str, sides)), requests=rng.randint(6, 16))
  return dict(kind=kind, side=between(8, 62), **material)  # spmv, energy


# ---- inputs ---------------------------------------------------------------------------


@functools.lru_cache(maxsize=4)
def _cube_at_rest(side):
  return scenes.fem_cube(side, noise=0.0)


def _cube(case, seed):
  """The cube of the case, its positions drawn from the seed."""
  pinned, free = scenes.fem_positions(case["side"], noise=case["noise"], seed=seed)
  mu, lam = scenes.lame(case["young"], case["poisson"])
  return dataclasses.replace(_cube_at_rest(case["side"]), pinned_position=pinned, free_position=free, mu=mu, lam=lam)


def _cloth(case, seed):
  """Cloth over the obstacle at the start of the step, and the positions it
  has moved to since (so the lagged friction slides)."""
  rng = np.random.default_rng([seed, 1])
  if case["kind"] == "dynamic":  # one set of active pairs (so of stored blocks), distances from the seed
    cc = scenes.cloth_contact(case["side"], case["pairs"], seed=0)
    obstacle = cc.obstacle.copy()
    obstacle[:, 1] = -np.sqrt(rng.uniform(0.1, 1.0, size=len(obstacle)) * cc.dhat)
    cc = dataclasses.replace(cc, obstacle=obstacle)
  else:
    cc = scenes.cloth_contact(case["side"], case["pairs"], num_bodies=case.get("bodies", 0), seed=seed)
  return cc, cc.cloth_position + rng.normal(0.0, 1e-5, cc.cloth_position.shape)


def _dynamic_scene(cc, position, method):
  """Cloth with dynamic sets of point-triangle and edge-edge pairs (``dynamic_instances``)."""
  sc = make_scene("dynamic")
  body = sc.addMesh("cloth")
  obst = body.addPrimitive("obstacle", numInstances=len(cc.obstacle))
  opos = obst.addAttribute("position", rows=3, cols=1)
  opos.updateValue(cc.obstacle)
  cloth = body.addPrimitive("cloth", numInstances=len(cc.cloth_position))
  pos = cloth.addAttribute("position", rows=3, cols=1)
  pos.updateValue(position)
  rest = cloth.addConstant("rest_position", rows=3, cols=1)
  rest.updateValue(cc.cloth_rest)
  mass = cloth.addConstant("mass")
  mass.updateValue(cc.mass)
  old = cloth.addConstant("old_position", rows=3, cols=1)
  old.updateValue(cc.cloth_position)
  tri = body.addPrimitive("triangles", numInstances=len(cc.tris))
  tc = tri.addConnectivity("to_cloth", cloth, cc.tris.astype(np.uint32), 3)
  mem = tri.addAttribute("stvk", computed_attribute=E.stvk_membrane(
      tri.addAttribute("rest", through=tc, source=rest), tri.addAttribute("x", through=tc, source=pos),
      cc.mu, cc.lam, cc.thickness, cc.dt))
  allv = body.addPrimitiveUnion("all_vertices", [obst, cloth])
  apos = allv.addAttribute("position")
  barriers = []
  for name, conn, energy in (("pt", cc.pt, E.point_triangle), ("ee", cc.ee, E.edge_edge)):
    pairs = body.addPrimitive(name + "_pairs", numInstances=len(conn), isDynamic=True)
    c = pairs.addConnectivity("to_vertices", allv, conn, 4)
    barriers.append(pairs.addAttribute("barrier", computed_attribute=energy(
        pairs.addAttribute("x", through=c, source=apos), cc.dhat, cc.kappa)))
  kin = cloth.addAttribute("inertia", computed_attribute=E.inertia(old, None, cc.dt, pos, mass,
                                                                   gravity=(0.0, -9.8, 0.0)))
  sc.addEnergy(mem, projection_method=method)
  for bar in barriers:
    sc.addEnergy(bar, projection_method=method, dynamic_instances=True)
  sc.addEnergy(kin, projection_method=-1)
  sc.addMinimizeTarget([pos])
  return sc


def _requests(case, seed):
  """Newton-step requests over the case's sides, materials as in the streams
  of the benchmark, positions in pinned host memory."""
  sides = [int(s) for s in case["sides"].split(",")]
  rng = np.random.default_rng([seed, 2])
  return [serving.fem_request(sides[k % len(sides)], float(10 ** rng.uniform(4, 6)), float(rng.uniform(0.3, 0.45)),
                              0.01, seed * 1009 + k, tag=k) for k in range(case["requests"])]


def prepare(case, seed):
  kind = case["kind"]
  if kind == "serve":
    server = serving.NewtonServer(max_slots=16, tolerance=TOL)
    reqs = _requests(case, seed)
    server.reserve(reqs)
    return dict(case=case, server=server, requests=reqs)
  if kind in ("cloth_step", "contact"):
    cc, moved = _cloth(case, seed)
    sc, handles = scenes.cloth_contact_scene(cc, projection_method=case.get("method", 1))
    handles["position"].updateValue(moved)
  elif kind == "dynamic":
    sc, handles = _dynamic_scene(*_cloth(case, seed), case["method"]), {}
  else:
    method = case["method"] if kind == "compute" else 1
    sc, handles = scenes.fem_scene(_cube(case, seed), projection_method=method)
  state = dict(case=case, scene=sc)
  mz = sc.minimizer
  if kind in ("step", "cloth_step"):
    mz.setSolver("mas", mixed_spmv=case["mixed"], stop_rule="residual")
    sc.minimizeEnergy(tolerance=TOL, maxIterations=MAX_IT)  # builds the plans a program keeps over its steps
  elif kind in ("compute", "contact", "dynamic"):
    mz.computeNumericValue()
  elif kind == "solve":
    state["H"] = mz.computeNumericValue()
    state["solver"] = make_solver(case["method"], stop_rule="residual")
    _solve(state)
  elif kind == "spmv":
    state["H"] = H = mz.computeNumericValue()
    rng = np.random.default_rng([seed, 3])
    state["x"] = vector(H.rows, torch.from_numpy(rng.normal(size=H.rows)).cuda())
    H.spmv(state["x"])
  elif kind == "energy":
    sc.computeTotalEnergy()
  elif kind == "shape":
    snh = handles["snh"]
    free_rest = resolve_leaf_children(snh.expr.rest.source)[0][-1]
    J = differentiator().diff2([snh], [handles["free_position"]], [free_rest])
    n = handles["free_position"].correspondance.numInstances * 3
    rng = np.random.default_rng([seed, 3])
    state.update(J=J, x=vector(n, torch.from_numpy(rng.normal(size=n)).cuda()),
                 y=vector(n, torch.from_numpy(rng.normal(size=n)).cuda()))
    J.compute()
  torch.cuda.synchronize()
  return state


def _solve(state):
  H, s = state["H"], state["solver"]
  s.computeSolution(H, H.gradient, None, tolerance=TOL, maxIterations=MAX_IT, zero_initial_guess=True)
  return s.solution


def run(state):
  kind = state["case"]["kind"]
  if kind == "serve":
    done = state["server"].run(state["requests"])
    return [r.solution for r in sorted(done, key=lambda r: r.tag)]
  sc = state["scene"]
  if kind in ("step", "cloth_step"):
    segments = sc.minimizeEnergy(tolerance=TOL, maxIterations=MAX_IT)
    return list(segments) + [sc.gradient]
  if kind in ("compute", "contact"):
    H = sc.minimizer.computeNumericValue()
    return [H.gradient.value, H.blocks_flattened]
  if kind == "dynamic":
    H = sc.minimizer.computeNumericValue()
    return [H.gradient.value, H.blocks_flattened, H.blocks_flattened_dynamic, H.block_positions_dynamic]
  if kind == "solve":
    return _solve(state)
  if kind == "spmv":
    return state["H"].spmv(state["x"]).value
  if kind == "energy":
    return sc.computeTotalEnergy()
  J = state["J"].compute()
  return [J.blocks_flattened, J.spmv(state["x"]).value, J.spmv(state["y"], transpose=True).value]


# ---- work and tolerances --------------------------------------------------------------


def _fem_counts(n):
  """Free vertices, tetrahedra, stored upper blocks of an n^3 cube with its
  z = 0 layer pinned."""
  m = n - 1
  nv = n * n * m
  edges = 2 * (n - 1) * n * m + n * n * (m - 1) + (n - 1) ** 2 * m + 2 * (n - 1) * n * (m - 1) + (n - 1) ** 2 * (m - 1)
  return nv, 6 * (n - 1) ** 3, nv + edges


def _cloth_counts(case):
  """Cloth vertices, elements and stored blocks (own and bending edges)."""
  n = case["side"]
  nv, tris, bend = n * n, 2 * (n - 1) ** 2, 0 if case["kind"] == "dynamic" else 3 * n * n
  return nv, tris + bend + case["pairs"], 7 * nv if bend else 4 * nv


def work(case):
  kind = case["kind"]
  if kind == "serve":
    sides = [int(s) for s in case["sides"].split(",")]
    out = {"bytes": 0, "flops": 0}
    for k in range(case["requests"]):
      nv, nt, nb = _fem_counts(sides[k % len(sides)])
      out["bytes"] += 8 * 3 * (nv + sides[k % len(sides)] ** 3)
      out["flops"] += 3000 * nt + 40 * 36 * nb
    return out
  if kind in ("cloth_step", "contact", "dynamic"):
    nv, ne, nb = _cloth_counts(case)
    if kind == "cloth_step":
      return {"bytes": 8 * 9 * nv + 16 * ne, "flops": 4000 * ne + 300 * 36 * nb}
    return {"bytes": 8 * 9 * nv + 16 * ne + 72 * nb, "flops": 4000 * ne}
  nv, nt, nb = _fem_counts(case["side"])
  nall = case["side"] ** 3
  if kind == "step":
    return {"bytes": 48 * nall + 16 * nt + 2 * 24 * nv, "flops": 3000 * nt + 45 * 36 * nb}
  if kind == "compute":
    return {"bytes": 48 * nall + 16 * nt + 24 * nv + 72 * nb, "flops": 3000 * nt}
  if kind == "solve":
    return {"bytes": 72 * nb + 2 * 24 * nv, "flops": (50 if case["method"] == "mas" else 250) * 36 * nb}
  if kind == "spmv":
    return {"bytes": 72 * nb + 4 * nb + 2 * 24 * nv, "flops": 36 * nb}
  if kind == "energy":
    return {"bytes": 48 * nall + 16 * nt + 24 * nv, "flops": 120 * nt}
  return {"bytes": 48 * nall + 16 * nt + 2 * 72 * nb + 4 * 24 * nv, "flops": 5000 * nt}


def tolerance(case):
  kind = case["kind"]
  # solutions: two solves that meet the relative residual of 1e-6 differ by
  # up to the condition number times that; measured against a 1e-11 solve:
  # 1.5e-5 (cubes), 1.5e-3 (the bodies' matrices over stiff contacts)
  if kind == "cloth_step":
    return {"rel": 8e-3}
  if kind in ("step", "solve", "serve"):
    return {"rel": 1e-4}
  # FP64 sums in another order give up to 2e-14 (gradients that nearly
  # cancel); eigenvalue iterations of 9x9 or 12x12 matrices in another order
  # about 2.5e-13
  return {"rel": 1e-12}


# ---- 64-bit results by plain torch ----------------------------------------------------

DEV = "cuda" if torch.cuda.is_available() else "cpu"
warnings.filterwarnings("ignore", message="Sparse ")


def _t(a, dtype=torch.float64):
  return torch.as_tensor(np.asarray(a), device=DEV).to(dtype)


def _det(a, b, c):
  return (a * torch.linalg.cross(b, c)).sum()


def _snh(x, r, mu, lam, dt):
  e, d = r[1:] - r[:1], x[1:] - x[:1]
  det = _det(e[0], e[1], e[2])
  inv = torch.stack([torch.linalg.cross(e[1], e[2]), torch.linalg.cross(e[2], e[0]),
                     torch.linalg.cross(e[0], e[1])]) / det
  f = d.T @ inv
  ic, j = (f * f).sum(), _det(f[:, 0], f[:, 1], f[:, 2])
  alpha = 1.0 + 0.75 * mu / lam
  return det / 6.0 * dt * dt * (0.5 * mu * (ic - 3.0) - 0.5 * mu * torch.log(ic + 1.0) + 0.5 * lam * (j - alpha) ** 2)


def _barrier(d, dhat, kappa):
  return kappa * (d - dhat) ** 2 * torch.log(d / dhat) ** 2


def _point_triangle(x, r, dhat, kappa):
  b = torch.linalg.cross(x[2] - x[1], x[3] - x[1])
  return _barrier(((x[0] - x[1]) * b).sum() ** 2 / (b * b).sum(), dhat, kappa)


def _edge_edge(x, r, dhat, kappa):
  b = torch.linalg.cross(x[1] - x[0], x[3] - x[2])
  return _barrier(((x[2] - x[0]) * b).sum() ** 2 / (b * b).sum(), dhat, kappa)


def _dihedral(q):
  n0 = torch.linalg.cross(q[0] - q[2], q[1] - q[2])
  n1 = torch.linalg.cross(q[1] - q[3], q[0] - q[3])
  axis = q[1] - q[0]
  num = (torch.linalg.cross(n0, n1) * axis).sum() / axis.norm()
  return 2.0 * torch.atan2(num, (n0 * n1).sum() + n0.norm() * n1.norm())


def _bending(x, r, kb, dt):
  return kb * (r[1] - r[0]).norm() * dt * dt * (_dihedral(x) - _dihedral(r)) ** 2


def _stvk(x, r, mu, lam, h, dt):
  # StVK is isotropic: any orthonormal frame of the rest triangle will do
  e1, e2 = r[1] - r[0], r[2] - r[0]
  u = e1 / e1.norm()
  n = torch.linalg.cross(e1, e2)
  w = torch.linalg.cross(n / n.norm(), u)
  m00, m01, m11 = e1.norm(), (e2 * u).sum(), (e2 * w).sum()
  f0 = (x[1] - x[0]) / m00
  f1 = ((x[2] - x[0]) - m01 * f0) / m11
  a, b, c = 0.5 * ((f0 * f0).sum() - 1.0), 0.5 * ((f1 * f1).sum() - 1.0), 0.5 * (f0 * f1).sum()
  return h * 0.5 * n.norm() * dt * dt * (mu * (a * a + b * b + 2.0 * c * c) + 0.5 * lam * (a + b) ** 2)


def _friction(x, r, q, fdhat, dt, rate):
  d = x - r
  rel = d[0] - (d[1] + q[0] * (d[2] - d[1]) + q[1] * (d[3] - d[1]))
  u0, u1 = (q[2:5] * rel).sum(), (q[5:8] * rel).sum()
  y2 = u0 * u0 + u1 * u1
  y = torch.sqrt(y2 + 1e-16)
  eps = fdhat ** 0.5 * dt
  phi = torch.where(y2 > fdhat * dt * dt, y, y2 / eps + eps / 3.0 - y2 * y / (3.0 * eps * eps))
  return rate * q[8] * phi


def _orthogonality(a, k):
  m = a.reshape(3, 3)
  d = m.T @ m - torch.eye(3, dtype=m.dtype, device=m.device)
  return 0.5 * k * (d * d).sum()


def _project(h, method):
  if method < 1:
    return h
  out = []
  for part in h.split(8192):
    w, v = torch.linalg.eigh(part)
    w = torch.where(w < 0, -w if method == 1 else torch.zeros_like(w), w)
    out.append((v * w[:, None, :]) @ v.transpose(1, 2))
  return torch.cat(out)


def _local(energy, shape, arrays, params, method):
  """Gradients and projected Hessians [n, k], [n, k, k] of a batch of elements."""
  def flat(z, *rest):
    return energy(z.reshape(shape), *rest, *params)
  x = arrays[0].reshape(len(arrays[0]), -1)
  both = torch.func.vmap(lambda *a: (torch.func.grad(flat)(*a), torch.func.hessian(flat)(*a)), chunk_size=200_000)
  g, h = both(x, *arrays[1:])
  return g, _project(h, method)


class _System:
  """Element terms over an extended vector [vertex coordinates, A matrices];
  the unknowns enter it through the sparse map ``lift`` (None: the free
  coordinates are the tail of the vector from ``first``)."""

  def __init__(self, size, first=0, lift=None):
    self.size, self.first, self.lift, self.terms = size, first, lift, []
    self.lift_t = None if lift is None else lift.t().to_sparse_csr()
    self.lift = None if lift is None else lift.to_sparse_csr()

  def add(self, idx, g, h):
    self.terms.append((idx, g, h))

  def up(self, q):
    if self.lift is not None:
      return self.lift @ q
    return torch.cat([q.new_zeros(self.first), q])

  def down(self, e):
    return self.lift_t @ e if self.lift is not None else e[self.first:]

  def gradient(self):
    e = torch.zeros(self.size, dtype=torch.float64, device=DEV)
    for idx, g, _ in self.terms:
      e.index_add_(0, idx.reshape(-1), g.reshape(-1))
    return self.down(e)

  def product(self, q):
    e, x = torch.zeros(self.size, dtype=torch.float64, device=DEV), self.up(q)
    for idx, _, h in self.terms:
      e.index_add_(0, idx.reshape(-1), torch.bmm(h, x[idx].unsqueeze(2)).reshape(-1))
    return self.down(e)

  def solve(self, g):
    e = torch.zeros(self.size, dtype=torch.float64, device=DEV)
    for idx, _, h in self.terms:
      e.index_add_(0, idx.reshape(-1), torch.diagonal(h, dim1=1, dim2=2).reshape(-1))
    if self.lift is None:
      diag = self.down(e)
    else:
      sq = torch.sparse_csr_tensor(self.lift_t.crow_indices(), self.lift_t.col_indices(), self.lift_t.values() ** 2,
                                   self.lift_t.shape)
      diag = sq @ e
    x, r = torch.zeros_like(g), g.clone()
    z = r / diag
    p, rz, stop = z.clone(), torch.dot(r, z), 1e-11 * float(g.norm())
    for it in range(20_000):
      q = self.product(p)
      alpha = rz / torch.dot(p, q)
      x += alpha * p
      r -= alpha * q
      if it % 20 == 0 and float(r.norm()) <= stop:
        break
      z = r / diag
      rz, old = torch.dot(r, z), rz
      p = z + (rz / old) * p
    return x

  def blocks(self, terms=None):
    """Upper 3x3 blocks sorted by (row, column) of the free coordinates."""
    n = self.size - self.first
    keys, vals = [], []
    for idx, _, h in self.terms if terms is None else terms:
      k = idx.shape[1] // 3
      b = h.reshape(len(h), k, 3, k, 3)
      v = idx[:, ::3] - self.first
      for i in range(k):
        for j in range(i, k):
          ok = (v[:, i] >= 0) & (v[:, j] >= 0)
          r, c, blk = v[ok, i], v[ok, j], b[ok][:, i, :, j, :]
          flip = (r > c)[:, None, None]
          keys.append(torch.minimum(r, c) * n + torch.maximum(r, c))
          vals.append(torch.where(flip, blk.transpose(1, 2), blk).reshape(-1, 9))
    key, inv = torch.unique(torch.cat(keys), return_inverse=True)
    out = torch.zeros((len(key), 9), dtype=torch.float64, device=DEV)
    out.index_add_(0, inv, torch.cat(vals))
    return key, out.reshape(-1)


def _coords(conn):
  c = _t(conn.astype(np.int64), torch.int64)
  return (3 * c[:, :, None] + torch.arange(3, device=DEV)).reshape(len(c), -1)


def _inertia(sys, vertices, x, target, mass):
  idx = _coords(vertices[:, None])
  sys.add(idx, _t(mass)[:, None] * _t(x - target), _t(mass)[:, None, None] * torch.eye(3, dtype=torch.float64, device=DEV))


def _fem_system(cube, method):
  x, r = _t(cube.positions_all()), _t(cube.rest_all())
  sys = _System(x.numel(), first=3 * cube.pinned_count)
  t = _t(cube.tets.astype(np.int64), torch.int64)
  g, h = _local(_snh, (4, 3), (x[t], r[t]), (cube.mu, cube.lam, cube.dt), method)
  sys.add(_coords(cube.tets), g, h)
  free = cube.pinned_count + np.arange(cube.free_count)
  _inertia(sys, free, cube.free_position, cube.x_tilde(), cube.mass)
  return sys


def _cloth_system(cc, moved, method, dynamic=False):
  """Vertices in the order [obstacle, cloth] or, with bodies, [obstacle,
  cloth, bodies] followed by the bodies' A."""
  no, nc = len(cc.obstacle), len(cc.cloth_position)
  points, lift = [cc.obstacle, moved], None
  bodies = cc.bodies
  if bodies is not None:
    points.append(bodies.positions())
    nb, nv = bodies.num_bodies, len(bodies.rest)
    b0 = 3 * (no + nc)
    v, vb = np.arange(nv), bodies.vertex_body
    rows, cols, vals = [3 * no + np.arange(3 * nc)], [np.arange(3 * nc)], [np.ones(3 * nc)]
    for k in range(3):
      for c in range(3):
        rows.append(b0 + 3 * v + k)
        cols.append(3 * nc + 9 * vb + 3 * k + c)
        vals.append(bodies.rest[:, c])
      rows.append(b0 + 3 * v + k)
      cols.append(3 * nc + 9 * nb + 3 * vb + k)
      vals.append(np.ones(nv))
    a0 = b0 + 3 * nv
    rows.append(a0 + np.arange(9 * nb))
    cols.append(3 * nc + np.arange(9 * nb))
    vals.append(np.ones(9 * nb))
    lift = torch.sparse_coo_tensor(torch.stack([_t(np.concatenate(rows), torch.int64), _t(np.concatenate(cols), torch.int64)]),
                                   _t(np.concatenate(vals)), (a0 + 9 * nb, 3 * nc + 12 * nb)).coalesce()
    sys = _System(a0 + 9 * nb, lift=lift)
  else:
    sys = _System(3 * (no + nc), first=3 * no)
  x = _t(np.concatenate(points))

  def term(energy, conn, extra, params, proj=method):
    c = _t(conn.astype(np.int64), torch.int64)
    k = conn.shape[1]
    sys.add(_coords(conn), *_local(energy, (k, 3), (x[c], *extra), params, proj))

  rest = _t(cc.cloth_rest)
  term(_stvk, cc.tris + no, (rest[_t(cc.tris, torch.int64)],), (cc.mu, cc.lam, cc.thickness, cc.dt))
  if not dynamic:
    term(_bending, cc.bend + no, (rest[_t(cc.bend, torch.int64)],), (cc.bend_stiff, cc.dt))
  pt = cc.pt.astype(np.int64)
  if len(pt):
    term(_point_triangle, pt, (x[_t(pt, torch.int64)],), (cc.dhat, cc.kappa))
    if not dynamic:
      old = _t(np.concatenate([cc.obstacle, cc.cloth_position]))
      term(_friction, pt, (old[_t(pt, torch.int64)], _t(cc.lagged)), (cc.fdhat, cc.dt, cc.friction))
  if len(cc.ee):
    term(_edge_edge, cc.ee, (x[_t(cc.ee.astype(np.int64), torch.int64)],), (cc.dhat, cc.kappa))
  gravity = np.array([0.0, -9.8, 0.0]) * cc.dt * cc.dt
  _inertia(sys, no + np.arange(nc), moved, cc.cloth_position + gravity, cc.mass)
  if bodies is not None:
    if len(cc.body_pt):
      # its union is [cloth, bodies, obstacle]
      u = cc.body_pt.astype(np.int64)
      conn = np.where(u < nc + nv, u + no, u - (nc + nv))
      term(_point_triangle, conn, (x[_t(conn, torch.int64)],), (cc.dhat, cc.kappa))
    p = bodies.positions()
    target = p + bodies.velocity * cc.dt + bodies.gravity[None] * cc.dt * cc.dt
    _inertia(sys, no + nc + v, p, target, bodies.mass)
    g, h = _local(_orthogonality, (9,), (_t(bodies.affine),), (bodies.stiffness,), 2)
    sys.add(a0 + torch.arange(9 * nb, device=DEV).reshape(nb, 9), g, h)
  return sys


def _shape(case, seed):
  cube = _cube(case, seed)
  x, r = _t(cube.positions_all()), _t(cube.rest_all())
  t = _t(cube.tets.astype(np.int64), torch.int64)

  def e(z, w):
    return _snh(z.reshape(4, 3), w.reshape(4, 3), cube.mu, cube.lam, cube.dt)
  mixed = torch.func.vmap(torch.func.jacfwd(torch.func.grad(e), argnums=1), chunk_size=200_000)
  h = mixed(x[t].reshape(-1, 12), r[t].reshape(-1, 12)).reshape(-1, 4, 3, 4, 3)
  v, n = t - cube.pinned_count, 3 * cube.free_count
  keys, vals = [], []
  for i in range(4):
    for j in range(4):
      ok = (v[:, i] >= 0) & (v[:, j] >= 0)
      keys.append(3 * v[ok, i] * n + 3 * v[ok, j])
      vals.append(h[ok][:, i, :, j, :].reshape(-1, 9))
  key, inv = torch.unique(torch.cat(keys), return_inverse=True)
  blocks = torch.zeros((len(key), 9), dtype=torch.float64, device=DEV).index_add_(0, inv, torch.cat(vals))
  rng = np.random.default_rng([seed, 3])
  a, b = _t(rng.normal(size=n)).reshape(-1, 3), _t(rng.normal(size=n)).reshape(-1, 3)
  row, col, m = key // n // 3, key % n // 3, blocks.reshape(-1, 3, 3)
  jx = torch.zeros_like(a).index_add_(0, row, torch.bmm(m, a[col].unsqueeze(2)).squeeze(2))
  jty = torch.zeros_like(b).index_add_(0, col, torch.bmm(m.transpose(1, 2), b[row].unsqueeze(2)).squeeze(2))
  return [blocks.reshape(-1), jx.reshape(-1), jty.reshape(-1)]


def exact(case, seed):
  kind = case["kind"]
  if kind == "serve":
    out = []
    for k, r in enumerate(_requests(case, seed)):
      pinned, free = scenes.fem_positions(r.side, noise=0.01, seed=seed * 1009 + k)
      cube = dataclasses.replace(_cube_at_rest(r.side), pinned_position=pinned, free_position=free, mu=r.mu, lam=r.lam)
      sys = _fem_system(cube, 1)
      out.append(sys.solve(sys.gradient()).cpu().numpy())
    return out
  if kind == "shape":
    return _shape(case, seed)
  if kind in ("cloth_step", "contact"):
    cc, moved = _cloth(case, seed)
    sys = _cloth_system(cc, moved, case.get("method", 1))
    g = sys.gradient()
    if kind == "contact":
      return [g, sys.blocks()[1]]
    x = sys.solve(g)
    n = 3 * len(cc.cloth_position)
    if cc.bodies is None:
      return [x, g]
    nb = cc.bodies.num_bodies
    return [x[:n], x[n:n + 9 * nb], x[n + 9 * nb:], g]
  if kind == "dynamic":
    cc, moved = _cloth(case, seed)
    sys = _cloth_system(cc, moved, case["method"], dynamic=True)
    key, values = sys.blocks(sys.terms[1:3])  # the terms: membrane, point-triangle, edge-edge, inertia
    n = 3 * len(cc.cloth_position)
    positions = torch.stack([key // n, key % n], dim=1).reshape(-1).to(torch.int32)
    return [sys.gradient(), sys.blocks([sys.terms[0], sys.terms[3]])[1], values, positions]
  cube = _cube(case, seed)
  if kind == "energy":
    x, r, t = _t(cube.positions_all()), _t(cube.rest_all()), _t(cube.tets.astype(np.int64), torch.int64)
    e = torch.func.vmap(lambda a, b: _snh(a, b, cube.mu, cube.lam, cube.dt), chunk_size=200_000)(x[t], r[t]).sum()
    d = cube.free_position - cube.x_tilde()
    return float(e) + float(np.sum(0.5 * cube.mass * np.sum(d * d, axis=1)))
  sys = _fem_system(cube, case["method"] if kind == "compute" else 1)
  g = sys.gradient()
  if kind == "compute":
    return [g, sys.blocks()[1]]
  if kind == "spmv":
    rng = np.random.default_rng([seed, 3])
    return sys.product(_t(rng.normal(size=len(g))))
  if kind == "solve":
    return sys.solve(g)
  return [sys.solve(g), g]
