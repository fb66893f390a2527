"""The MAS-PCG loop as a graph of kernels, the form of systems beyond the
one-kernel loop's sizes, at sizes that a host check can follow: each of its
products (FP64 and FP32 row plan, tiled, streamed; one block set and two) and a
one-level hierarchy.  Each solution's true relative residual is taken in FP64 on
the host; the bound is the solve's own (a tenth more covers the drift of the
recursive residual)."""

import numpy as np
import pytest

from tests import test_gpu_long_rows as long_rows
from tests.test_gpu_loop import residual
from yasps_b200 import scenes

pytestmark = pytest.mark.gpu


def cube(side, mixed, one_kernel=False, **options):
  sc, _ = scenes.fem_scene(scenes.fem_cube(side, noise=0.01, seed=side))
  solver = sc.minimizer.setSolver("mas", mixed_spmv=mixed, stop_rule="residual", **options)
  solver.implementation.one_kernel_loop = one_kernel
  return sc, solver


@pytest.mark.parametrize("product", ["fp64", "tiled", "streamed"])
@pytest.mark.parametrize("side,options", [(3, {}), (12, {}), (20, {}),
                                          (12, dict(max_levels=1, global_coarse_domain=False))])
def test_cube_solutions(side, options, product):
  sc, solver = cube(side, product != "fp64", **options)
  H = sc.minimizer.computeNumericValue()
  (bs,) = H.block_sets
  solves = []
  for _ in range(2):
    if product == "tiled":
      bs.stream = False
    code = solver.computeSolution(H, H.gradient, None, tolerance=1e-6, maxIterations=2000, zero_initial_guess=True)
    assert code == 0 and solver.statistics["converged"]
    solves.append(solver.solution.cpu().numpy().copy())
  assert residual(H, solves[0]) <= 1.1e-6
  assert np.array_equal(*solves)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("side", [14, 72])
def test_two_block_sets(side, mixed):
  s = long_rows.Scene(side, mixed)
  s.solver.implementation.one_kernel_loop = False
  for pairs in (s.path(), s.hub(9)):
    H = s.compute(pairs)
    assert long_rows.residual(H, s.solve(H).cpu().numpy()) <= 1.1e-6


def test_first_size_beyond_the_one_kernel_loop():
  """A 49^3 cube (115,248 variables) runs the graph of kernels by itself."""
  solutions = []
  for one_kernel in (True, False):
    sc, _ = cube(49, True, one_kernel)
    solutions.append(sc.minimizeEnergy(tolerance=1e-6, maxIterations=2000)[0].cpu().numpy())
  assert residual(sc.minimizer.activeHessian(), solutions[0]) <= 1.1e-6
  assert np.array_equal(*solutions)
