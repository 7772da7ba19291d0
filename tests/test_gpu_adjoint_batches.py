"""The dense backward's gradient copies: groups of 128 pairs take them in turn, so every pair lands in the batch its
number gives, whatever blocks walk it; sizes around a chunk, a couple, a group, every block count an SM."""

import numpy as np
import pytest
import torch

from optlab_b200 import workloads
from optlab_b200.adjoint import AdjointPlan

pytestmark = pytest.mark.gpu

BATCHES = 32


def _expected(n_pairs, precision, names):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    copies = min(-(-n_pairs // 128), sms * (3 if precision == "fp32" else 2 if names <= 2 else 1))
    group = np.arange(n_pairs) // 128
    return np.bincount(group % copies % BATCHES, minlength=BATCHES)


# (60003: the one-round launch of seven blocks an SM; 131072 + 65: several passes a block and a ragged group)
@pytest.mark.parametrize("n_pairs", [2, 33, 65, 129, 4097, 60003, 131137])
@pytest.mark.parametrize("names", [1, 3, 4])
def test_every_pair_falls_in_its_batch_and_the_copies_add_up(n_pairs, names):
    c, rho = [0.03, 0.045, 0.06, 0.05][:names], [-0.7, -0.55, -0.4, -0.5][:names]
    w = workloads.worst_of(n_paths=2 * n_pairs, years=1.0, steps_per_year=12, n_names=names, c=c, rho=rho, n_exp=4,
                           n_x=33)
    with AdjointPlan(w.held, 0.005, "fp32", checkpoint=1) as dense, \
            AdjointPlan(w.held, 0.005, "fp32", checkpoint=4) as sparse:
        dense.run()
        sparse.run()
        assert np.array_equal(dense.batch_pairs.cpu().numpy(), _expected(n_pairs, "fp32", names))
        gd, gs = dense.gradient.cpu().numpy(), sparse.gradient.cpu().numpy()
    # twelve float steps: the two backwards' noise terms agree to some 1e-5 of a weight, the sums of some 1e5 of them to
    # less of the largest entry
    assert np.abs(gd - gs).max() <= 2e-4 * np.abs(gs).max()
