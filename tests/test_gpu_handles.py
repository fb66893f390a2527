"""Handles of different sizes alive at once: the limit of a kernel's dynamic
shared memory belongs to the process, so a handle of small domains must leave
room for the launches of a larger one made before it."""

import pytest

from tests.test_gpu_loop import residual
from yasps_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("side", [9, 20])  # 96-DoF domains: one a CTA, and warps over many
def test_small_handle_after_a_large_one(side, mixed):
  def make(n):
    sc, _ = scenes.fem_scene(scenes.fem_cube(n, noise=0.01, seed=n))
    sc.minimizer.setSolver("mas", mixed_spmv=mixed, stop_rule="residual")
    return sc

  def solve(sc):
    x = sc.minimizeEnergy(tolerance=1e-6, maxIterations=500)[0]
    assert residual(sc.minimizer.activeHessian(), x.cpu().numpy()) <= 1.1e-6
    return x.clone()

  large = make(side)
  first = solve(large)
  dofs = large.minimizer.linearSolver.implementation._tables.max_domain_dofs
  small = make(3)
  solve(small)
  assert small.minimizer.linearSolver.implementation._tables.max_domain_dofs < dofs
  assert bool((solve(large) == first).all())
