"""The node vegas' standard errors for counts of pairs that do not fill every batch (of 128 pairs each): they measure the
vegas' spread over independent seeds, by the node kernels and through torch, and are defined for a single batch."""

import numpy as np
import pytest

from optlab_b200 import workloads
from optlab_b200.adjoint import AdjointPlan, VegaNodes, autocall_greeks

pytestmark = pytest.mark.gpu


class ThroughTorch(VegaNodes):
    """(the node kernels take VegaNodes themselves alone)"""


def _greeks(n_pairs, seed, nodes_type, checkpoint):
    w = workloads.worst_of(n_paths=2 * n_pairs, seed=seed, years=1.0, steps_per_year=12, n_names=2, c=[0.03, 0.045],
                           rho=[-0.7, -0.55], n_exp=4, n_x=33)
    nodes = nodes_type(w.row_name, w.row_T, w.row_lo, w.row_inv_dx, w.n_x, np.linspace(0.2, 1.0, 3),
                       np.linspace(-0.5, 0.25, 4))
    with AdjointPlan(w.held, 0.02, "fp32", checkpoint=checkpoint) as plan:
        return autocall_greeks(w.held, nodes, 0.02, "fp32", plan=plan)


@pytest.mark.parametrize("n_pairs,nodes_type,checkpoint", [
    (900, VegaNodes, 1),      # 8 batches of groups of 128 pairs
    (1500, VegaNodes, 1),     # groups of 32
    (2048, VegaNodes, 1),     # groups of 64
    (2048, VegaNodes, 4),     # the recomputing backward: 8 batches, one a block of 256 pairs
    (900, ThroughTorch, 1),
])
def test_vega_errors_measure_the_spread_over_seeds(n_pairs, nodes_type, checkpoint):
    seeds = 400
    runs = [_greeks(n_pairs, 1000 + s, nodes_type, checkpoint) for s in range(seeds)]
    spread = np.var([r["vega"] for r in runs], axis=0, ddof=1)
    told = np.mean([r["vega_se"] ** 2 for r in runs], axis=0)
    # A variance from 400 normal values is known to a relative sqrt(2 / 399) = 7 %, however the nodes depend on each
    # other, and the mean of 400 estimates of 7 and more degrees of freedom to sqrt(2 / 2800) = 3 %: four deviations.
    # (Counting the empty batches makes the ratio (k - 1) / 31 with k batches: 0.23 at 8, 0.35 at 12, 0.48 at 16.)
    ratio = told.sum() / spread.sum()
    assert abs(np.log(ratio)) < 4 * np.hypot(np.sqrt(2 / 399), np.sqrt(2 / 2800)), ratio


@pytest.mark.parametrize("nodes_type", [VegaNodes, ThroughTorch])
def test_a_single_batch_has_no_error_to_tell(nodes_type):
    g = _greeks(100, 5, nodes_type, 1)
    assert np.any(g["vega"] != 0) and np.all(g["vega_se"] == 0)
