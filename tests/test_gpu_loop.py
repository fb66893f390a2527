"""The one-kernel MAS-PCG loop (``mas_pcg_loop``) at the sizes where it can go
wrong: one domain and one CTA, a domain a CTA (the wide form, more CTAs than
the row count alone would take), the first sizes past it, and rows long enough
to be split over warps (affine bodies in contact).  Each solution's true
relative residual is taken in FP64 on the host; the bound is the solve's own
(the stop test of the FP64 loop runs on the recursive residual: a tenth more
covers its drift)."""

import numpy as np
import pytest
from scipy.sparse import coo_matrix

from yasps_b200 import scenes

pytestmark = pytest.mark.gpu


def residual(H, x):
  pos, val = H.blocks3()
  pos, val = pos.cpu().numpy().astype(np.int64).reshape(-1, 2), val.cpu().numpy().reshape(-1, 3, 3)
  r = (pos[:, 0, None, None] + np.arange(3)[None, :, None]) + np.zeros((1, 1, 3), dtype=np.int64)
  c = (pos[:, 1, None, None] + np.arange(3)[None, None, :]) + np.zeros((1, 3, 1), dtype=np.int64)
  off = pos[:, 0] != pos[:, 1]
  A = coo_matrix((np.concatenate([val.ravel(), val[off].ravel()]),
                  (np.concatenate([r.ravel(), c[off].ravel()]), np.concatenate([c.ravel(), r[off].ravel()]))),
                 shape=(H.rows, H.rows)).tocsr()
  g = H.gradient.value.cpu().numpy()
  return np.linalg.norm(g - A @ x) / np.linalg.norm(g)


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("side", [3, 4, 9, 17, 18, 20])
def test_cube_solutions(side, mixed):
  sc, _ = scenes.fem_scene(scenes.fem_cube(side, noise=0.01, seed=side))
  solver = sc.minimizer.setSolver("mas", mixed_spmv=mixed, stop_rule="residual")
  first = sc.minimizeEnergy(tolerance=1e-6, maxIterations=500)[0].clone()
  assert residual(sc.minimizer.activeHessian(), first.cpu().numpy()) <= 1.1e-6
  again = sc.minimizeEnergy(tolerance=1e-6, maxIterations=500)[0]
  assert bool((again == first).all())  # fixed order of every sum
  assert solver.statistics["converged"]


@pytest.mark.parametrize("mixed", [True, False])
def test_rows_split_over_warps(mixed):
  cc = scenes.cloth_contact(56, 1000, spacing=0.025, dhat=1e-2, num_bodies=1, body_subdivisions=4, seed=2)
  sc, _ = scenes.cloth_contact_scene(cc)
  sc.minimizer.setSolver("mas", mixed_spmv=mixed, stop_rule="residual")
  x = np.concatenate([s.cpu().numpy() for s in sc.minimizeEnergy(tolerance=1e-6, maxIterations=5000)])
  H = sc.minimizer.activeHessian()
  row_ptr = H.spmv_plan(H.block_sets[0])[0][:H.rows // 3 + 1].cpu().numpy()
  assert np.diff(row_ptr).max() > 128, "the scene must hold a row of more than one segment"
  assert residual(H, x) <= 1.1e-6
