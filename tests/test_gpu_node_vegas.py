"""The node kernels behind autocall_greeks against torch's contraction of the same run's gradients, over names, node
counts and table widths around a warp of strikes, a block of outputs and a chunk of cells; and what they do not take."""

import numpy as np
import pytest
import torch

from optlab_b200 import workloads
from optlab_b200.adjoint import AdjointPlan, VegaNodes, autocall_greeks

pytestmark = pytest.mark.gpu

EPS64 = np.finfo(float).eps


def _case(names, n_x, n_e, n_k, n_pairs=1500, **kw):
    c, rho = [0.03, 0.045, 0.06, 0.05][:names], [-0.7, -0.55, -0.4, -0.5][:names]
    w = workloads.worst_of(n_paths=2 * n_pairs, years=1.0, steps_per_year=12, n_names=names, c=c, rho=rho, n_exp=4,
                           n_x=n_x)
    nodes = VegaNodes(w.row_name, w.row_T, w.row_lo, w.row_inv_dx, w.n_x, np.linspace(0.2, 1.0, n_e),
                      np.linspace(-1.0, 0.5, n_k), **kw)
    s = w.held.struct
    table = np.ctypeslib.as_array(s.table, shape=(s.n_rows * s.n_x,)).reshape(s.n_rows, s.n_x)
    return w, nodes, torch.tensor(table, dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("names,n_x,n_e,n_k", [(1, 33, 2, 2), (2, 255, 3, 8), (3, 101, 10, 15), (4, 257, 5, 9),
                                               (1, 600, 4, 33)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_node_vegas_equal_the_contraction_of_the_gradients(names, n_x, n_e, n_k, precision):
    w, nodes, base = _case(names, n_x, n_e, n_k)
    with AdjointPlan(w.held, 0.005, precision) as plan:
        g = autocall_greeks(w.held, nodes, 0.005, precision, plan=plan)
        grads, pairs, mean_grad = plan.batch_grad, plan.batch_pairs, plan.gradient
    vega = nodes.contract(mean_grad, base).cpu().numpy()
    vb = nodes.contract_batches(grads / pairs.clamp(min=1.0)[:, None, None], base).cpu().numpy()
    size = nodes.contract_batches(grads.abs() / pairs.clamp(min=1.0)[:, None, None], base).cpu().numpy()
    p = pairs.cpu().numpy()[:, None, None, None] / pairs.sum().item()
    se = np.sqrt((p * (vb - (p * vb).sum(0)) ** 2).sum(0) * 32 / 31 / 32)
    # both sum the same products in their own order: a sum of m terms is within m roundings of their magnitudes' sum, and
    # a product carries a few; a batch mean that is off by d moves the standard error by at most d's own (weighted) size
    terms = base.numel() + 32 + 16
    bound = terms * EPS64 * (p * size).sum(0)
    assert g["vega"].shape == g["vega_se"].shape == nodes.shape
    assert np.all(np.abs(g["vega"] - vega) <= 2 * bound)
    assert np.all(np.abs(g["vega_se"] - se) <= 4 * terms * EPS64 * (np.sqrt((p * size**2).sum(0)) + se))


def test_other_nodes_go_through_torch_with_the_same_values():
    class Own(VegaNodes):
        pass

    w, nodes, base = _case(3, 101, 4, 5)
    own = Own(w.row_name, w.row_T, w.row_lo, w.row_inv_dx, w.n_x, nodes.node_T, nodes.node_k)
    with AdjointPlan(w.held, 0.005, "fp64") as plan:
        a = autocall_greeks(w.held, nodes, 0.005, "fp64", plan=plan)
        b = autocall_greeks(w.held, own, 0.005, "fp64", plan=plan)
        assert a["price"] == b["price"] and np.array_equal(a["delta"], b["delta"])
        # (the double backward's additions come in any order: a relative 1e-10 of the largest vega holds ample roundings)
        for k in ("vega", "vega_se"):
            assert np.abs(a[k] - b[k]).max() <= 1e-10 * np.abs(b[k]).max()
        with torch.no_grad(), pytest.raises(RuntimeError):
            autocall_greeks(w.held, nodes, 0.005, "fp64", plan=plan)
