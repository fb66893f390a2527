"""Level-2 domains of the one-kernel MAS-PCG loop dealt three to a CTA (more than
twelve of them) and one to a CTA.  Each solution's true relative residual is
taken in FP64 on the host; the bound is the solve's own (a tenth more covers the
drift of the recursive residual)."""

import numpy as np
import pytest

from tests.test_gpu_loop import residual
from yasps_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("side,bodies,grouped", [(112, 4, False), (256, 16, True)])
def test_level_two_domains(side, bodies, grouped, mixed):
  cc = scenes.cloth_contact(side, 3 * side * side, num_bodies=bodies)
  sc, _ = scenes.cloth_contact_scene(cc)
  solver = sc.minimizer.setSolver("mas", mixed_spmv=mixed, stop_rule="residual")
  first = np.concatenate([s.cpu().numpy() for s in sc.minimizeEnergy(tolerance=1e-6, maxIterations=5000)])
  domains = solver.statistics["domains_per_level"]
  assert (len(domains) > 2 and domains[2] > 12) == grouped, domains
  assert residual(sc.minimizer.activeHessian(), first) <= 1.1e-6
  again = np.concatenate([s.cpu().numpy() for s in sc.minimizeEnergy(tolerance=1e-6, maxIterations=5000)])
  assert np.array_equal(first, again)  # fixed order of every sum
