"""The float local-vol step on packed pairs of legs: tables from two points to more than the shared-memory stage holds,
narrow enough that paths run past both ends, against the FP64 oracle; and a variance that is not a number."""

import numpy as np
import pytest

from optlab_b200 import engine
from optlab_b200._abi import OB_MODEL_PATHS, OB_PRODUCT_AUTOCALL
from optlab_b200.requests import mc_request, paths_request, result_arrays

pytestmark = pytest.mark.gpu

STEPS = 43  # no multiple of any batch of steps


def _model(names, n_x):
    rng = np.random.default_rng(3)
    corr = np.full((names, names), 0.4) + 0.6 * np.eye(names)
    rows = (0.04 + 0.02 * np.cos(np.linspace(0, 2, n_x)))[None, :] * (1 + 0.2 * rng.random((STEPS, n_x)))
    return dict(dt=np.full(STEPS, 1 / 252), t0=np.arange(STEPS) / 252, root=np.linalg.cholesky(corr), kind=[1] * names,
                cvar=np.zeros(names), step_row=np.tile(np.arange(STEPS), names), lo=np.full(STEPS, -0.05),
                inv_dx=np.full(STEPS, (n_x - 1) / 0.08), table=rows, n_x=n_x, seed=99)


@pytest.mark.parametrize("n_x", [2, 17, 801])
@pytest.mark.parametrize("names", [1, 2, 3, 5])
def test_two_float_steps_match_the_oracle_at_every_table_size_and_past_its_ends(oracle, names, n_x):
    kw = dict(_model(names, n_x), obs_step=[1, 2], heston=np.tile([0.0, 1, 1, 0, 0], names), same=1,
              fwd=np.full((names, 2), 100.0), n_pairs=4097)
    kw |= dict(dt=kw["dt"][:2], t0=kw["t0"][:2], step_row=np.tile([0, 1], names), lo=np.full(STEPS, -0.02),
               inv_dx=np.full(STEPS, (n_x - 1) / 0.03))
    g, o = paths_request(**kw), paths_request(**kw)
    engine.paths(g, "fp32")
    oracle.paths(o)
    x = [np.log(next(a for a in h.keep if isinstance(a, np.ndarray) and a.ndim == 3) / 100.0) for h in (g, o)]
    assert x[1][:, 0].min() < -0.025 and x[1][:, 0].max() > 0.015  # the second step starts past both ends
    # One step: a normal of at most 6.7, off by at most 3e-6 of its radius (twice that through the root), on a
    # deviation of at most 0.017, and a variance off by the cell's weight (n_x 2^-23 intervals) and a few roundings;
    # the price's own rounding. The next step reads the variance at a point off by as much: the table's slope.
    sd, z = np.sqrt(kw["table"].max() / 252), 6.7
    rise = np.abs(np.diff(kw["table"], axis=1)).max()
    weight = rise * n_x * 2.0**-23 / (2 * kw["table"].min())
    one = sd * z * (2 * 3e-6 + weight + 5e-7) + 3e-7
    slope = rise * kw["inv_dx"][0] / (2 * kw["table"].min()) * sd * z
    err = [np.abs(x[0][:, k] - x[1][:, k]).max() for k in (0, 1)]
    assert err[0] <= one and err[1] <= one * (2 + slope), (err, one, slope)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("names", [1, 2])
def test_a_path_that_is_not_a_number_is_never_knocked_in(names, precision):
    kw = _model(names, 17)
    kw["table"] = kw["table"].copy()
    kw["table"][20:] = -1.0  # every path is NaN from step 21 on, after its low has passed the knock-in level
    log_fwd = np.zeros((names, STEPS + 1))
    log_fwd[:, 1:10] = -1.0
    obs = np.array([30, 37, STEPS])
    held = mc_request(model=OB_MODEL_PATHS, product=OB_PRODUCT_AUTOCALL, spot=np.full(names, 100.0), n_pairs=257,
                      log_fwd=log_fwd, obs_step=obs, obs_discount=[0.9, 0.8, 0.7], trigger=[1.0, 1.0, 0.0],
                      coupon_barrier=0.7, coupon=0.02, ki_barrier=0.6, put_strike=1.0, memory=1, ki_daily=1, **kw)
    price, _ = result_arrays(engine.mc_price(held, precision))
    assert price.tolist() == [0.7, 0.0, 0.0, 0.0]
