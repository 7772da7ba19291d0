"""The double dense backward's gradient copies, one or two an SM: counts of pairs that share them, in one pass of the
blocks and in several, against the recomputing backward."""

import numpy as np
import pytest
from test_gpu_adjoint_batches import _expected

from optlab_b200 import workloads
from optlab_b200.adjoint import AdjointPlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pairs", [65, 1500, 3001, 60003, 131137])
@pytest.mark.parametrize("names", [1, 3, 4])
def test_every_pair_falls_in_its_batch_and_the_double_copies_add_up(n_pairs, names):
    c, rho = [0.03, 0.045, 0.06, 0.05][:names], [-0.7, -0.55, -0.4, -0.5][:names]
    w = workloads.worst_of(n_paths=2 * n_pairs, years=1.0, steps_per_year=12, n_names=names, c=c, rho=rho, n_exp=4,
                           n_x=33)
    with AdjointPlan(w.held, 0.005, "fp64", checkpoint=1) as dense, \
            AdjointPlan(w.held, 0.005, "fp64", checkpoint=4) as sparse:
        dense.run()
        sparse.run()
        pairs = dense.batch_pairs.cpu().numpy()
        gd, gs = dense.gradient.cpu().numpy(), sparse.gradient.cpu().numpy()
    if 1024 <= n_pairs < 4096:  # groups of 64 or 32 pairs
        group = 64 if n_pairs >= 2048 else 32
        assert np.array_equal(pairs, np.bincount(np.arange(n_pairs) // group % 32, minlength=32))
    else:
        assert np.array_equal(pairs, _expected(n_pairs, "fp64", names))
    # the backwards recover or redraw each step's noise in double: some roundings a step, amplified at most some thousand
    # times where a step's variance is small (the bound that the Greeks of both are held to)
    assert np.abs(gd - gs).max() <= 1e-9 * np.abs(gs).max()
