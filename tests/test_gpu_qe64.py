"""The FP64 Heston QE kernel's own step and functions against the oracle, where they change over: variances that never
leave the quadratic branch, that mostly sit at zero, corrections that leave the short logarithm's range or have no
finite value, step counts around a batch and ragged pair counts."""

import numpy as np
import pytest

from optlab_b200 import engine
from optlab_b200._abi import OB_MODEL_HESTON_QE, OB_PRODUCT_AUTOCALL, OB_PRODUCT_LADDER
from optlab_b200.requests import mc_request, result_arrays

pytestmark = pytest.mark.gpu

HESTON = {
    "quadratic only": (0.09, 2.0, 0.09, 0.1, -0.5),
    "at zero": (0.01, 0.5, 0.01, 1.5, -0.9),
    "starts at zero": (0.0, 1.5, 0.04, 0.5, -0.7),
    "large positive correction": (0.5, 30.0, 0.6, 0.3, 0.95),
    "large negative correction": (0.4, 8.0, 0.5, 3.0, -0.95),
    "uncorrelated": (0.04, 1.5, 0.04, 0.5, 0.0),
}


def _request(heston, steps, n_pairs, T, product):
    kw = dict(model=OB_MODEL_HESTON_QE, dt=np.full(steps, T / steps), t0=np.arange(steps) * T / steps, spot=[100.0],
              n_pairs=n_pairs, first_pair=2**31 + 7, seed=2**40 + 11, heston=heston, r=0.03, q=0.01, product=product)
    if product == OB_PRODUCT_LADDER:
        kw |= dict(leg_type=[1, 2, 3, 1, 2], leg_strike=[90.0, 100.0, 110.0, 100.0, 100.0], leg_barrier=[0, 0, 0, 1, 4],
                   leg_level=[0, 0, 0, 140.0, 80.0], discount=0.97)
    else:
        obs = sorted({max(1, steps // 3), steps})
        kw |= dict(obs_step=obs, obs_discount=np.linspace(0.99, 0.95, len(obs)),
                   trigger=[1.0] * (len(obs) - 1) + [0.0], coupon_barrier=0.8, coupon=0.01, ki_barrier=0.7,
                   put_strike=1.0, memory=1, ki_daily=1)
    return mc_request(**kw)


@pytest.mark.parametrize("product", [OB_PRODUCT_LADDER, OB_PRODUCT_AUTOCALL], ids=["ladder", "autocall"])
@pytest.mark.parametrize("steps,n_pairs", [(1, 2), (3, 33), (4, 513), (63, 2049)])
@pytest.mark.parametrize("name", HESTON)
def test_the_fp64_step_matches_the_oracle(oracle, name, steps, n_pairs, product):
    # few long steps make the corrections large: a year in 1, 3 or 4 steps
    args = (HESTON[name], steps, n_pairs, 1.0 if steps < 10 else 0.25, product)
    got, want = engine.mc_price(_request(*args), "fp64"), oracle.mc_price(_request(*args))
    g, w = np.array(result_arrays(got)), np.array(result_arrays(want))
    # each step's functions are within an ulp or two (4e-16), a step's recursion amplifies them at most some hundred
    # times (the variance's square root near zero), and there are at most 63 steps
    assert np.all(np.abs(g[0] - w[0]) <= 1e-11 * np.maximum(np.abs(w[0]), 1.0)), (g[0], w[0])
    assert np.all(np.abs(g[1] - w[1]) <= 1e-9 * np.maximum(np.abs(w[1]), 1.0))
