"""Heston QE over thousands of steps: the specialised kernel, which stages four bytes a step, against the oracle and
against the generic kernel on either side of the counts where a whole record a step filled the stage."""

import numpy as np
import pytest

from optlab_b200 import engine
from optlab_b200._abi import OB_MODEL_HESTON_QE, OB_PRODUCT_AUTOCALL, OB_PRODUCT_LADDER
from optlab_b200.requests import mc_request, result_arrays

pytestmark = pytest.mark.gpu


def _request(steps, product):
    kw = dict(model=OB_MODEL_HESTON_QE, dt=np.full(steps, 1 / 252), t0=np.arange(steps) / 252, spot=[100.0], n_pairs=65,
              seed=77, heston=(0.04, 1.5, 0.04, 0.5, -0.7), r=0.02, q=0.01, product=product)
    if product == OB_PRODUCT_LADDER:
        kw |= dict(leg_type=[1, 2, 1], leg_strike=[90.0, 110.0, 100.0], leg_barrier=[0, 0, 1], leg_level=[0, 0, 900.0],
                   discount=0.6)
    else:
        obs = np.unique([1, steps // 4, steps // 2, steps - 1, steps])
        kw |= dict(obs_step=obs, obs_discount=np.linspace(0.99, 0.6, len(obs)), trigger=[9.0] * (len(obs) - 1) + [0.0],
                   coupon_barrier=0.5, coupon=0.01, ki_barrier=0.3, put_strike=1.0, memory=1, ki_daily=1)
    return mc_request(**kw)


@pytest.mark.parametrize("product", [OB_PRODUCT_LADDER, OB_PRODUCT_AUTOCALL], ids=["ladder", "autocall"])
@pytest.mark.parametrize("steps,precision", [(6300, "fp64"), (6804, "fp64"), (7500, "fp64"), (7500, "fp32")])
def test_thousands_of_qe_steps_match_the_oracle_and_the_generic_kernel(oracle, monkeypatch, steps, precision, product):
    got = np.array(result_arrays(engine.mc_price(_request(steps, product), precision)))
    want = np.array(result_arrays(oracle.mc_price(_request(steps, product))))
    monkeypatch.setenv("OPTLAB_B200_GENERIC", "1")
    plain = np.array(result_arrays(engine.mc_price(_request(steps, product), precision)))
    # A step moves the log by a few roundings of its terms, amplified at most some hundred times where the variance sits
    # near zero (1e-11 over 63 steps in test_gpu_qe64): at most in proportion to the steps. In float 2^29 times that,
    # capped by a payment's own size, would say nothing: there the two kernels' prices differ by the steps' roundings.
    if precision == "fp64":
        bound = 1e-11 * steps / 63
        assert np.all(np.abs(got[0] - want[0]) <= bound * np.maximum(np.abs(want[0]), 1.0)), (got[0], want[0])
    else:
        bound = steps * 2.0**-24 * 4
    assert np.all(np.abs(got[0] - plain[0]) <= bound * np.maximum(np.abs(plain[0]), 1.0)), (got[0], plain[0])
