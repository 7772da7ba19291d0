"""The float kernels for many pairs, which small counts no longer reach (fewer pairs put their legs on two lanes):
ladders of whole pairs and of streamed rows against the oracle and against the same pairs in small pieces, and
observations on the edges of an eight-step batch."""

import numpy as np
import pytest

from optlab_b200 import engine, workloads
from optlab_b200.requests import mc_request, result_arrays

pytestmark = pytest.mark.gpu

STEPS, YEARS = 126, 0.5
WHOLE, STREAMED = 40000, 30001  # 148 SMs: whole pairs from 35521 (two and three names) or 26049; rows streamed to 56831
SMALL = 4096


def _ladder(names, n_x, n_pairs, first_pair=0):
    corr = np.full((names, names), 0.6) + 0.4 * np.eye(names)
    dt, t0 = workloads.uniform_grid(YEARS, STEPS)
    # eight expiries of 120 points in the stage, or a row a step beyond it (0.8 MB)
    g = workloads.lv_grid(horizon=YEARS, n_exp=8 if n_x == 120 else STEPS, n_x=n_x)
    m = workloads.FlatMarket(100.0, 0.02, 0.01)
    return dict(model=0, dt=dt, t0=t0, spot=100.0 + 10 * np.arange(names), n_pairs=n_pairs, seed=17, kind=[1] * names,
                root=np.linalg.cholesky(corr), cvar=np.zeros(names), first_pair=first_pair,
                log_fwd=np.tile(m.log_fwd(np.concatenate([[0.0], t0 + dt])), (names, 1)),
                step_row=np.tile(g.row_of(t0), (names, 1)), lo=g.lo, inv_dx=g.inv_dx, table=g.rows, n_x=n_x,
                product=0, leg_type=[1, 1, 2, 3, 2, 1], leg_strike=[80.0, 100.0, 120.0, 100.0, 100.0, 100.0],
                leg_barrier=[0, 0, 0, 0, 4, 1], leg_level=[0, 0, 0, 0, 85.0, 125.0], discount=float(m.D(YEARS)))


CASES = [(1, 120, WHOLE), (2, 120, WHOLE), (3, 120, WHOLE), (1, 801, STREAMED), (1, 801, 60001), (3, 801, WHOLE)]


@pytest.mark.parametrize("names,n_x,n_pairs", CASES)
def test_float_ladders_match_the_oracle(oracle, names, n_x, n_pairs):
    kw = _ladder(names, n_x, n_pairs)
    got, _ = result_arrays(engine.mc_price(mc_request(**kw), "fp32"))
    want, se = result_arrays(oracle.mc_price(mc_request(**kw)))
    # The same normals: a step's is off by at most 3e-6 of a radius of at most 6.7 (twice that through the root), its
    # variance by the cell's weight (n_x 2^-23 intervals) and a few roundings. All of a path's steps off by that in one
    # direction make some eight times what a typical draw's add up to, which holds the feedback of the table's slope.
    var = kw["table"]
    weight = np.abs(np.diff(var, axis=1)).max() * n_x * 2.0**-23 / (2 * var.min())
    step = np.sqrt(var.max() * YEARS / STEPS) * 6.7 * (2 * 3e-6 + weight + 5e-7) + 3e-7
    paid = 120.0 * STEPS * step
    plain = [0, 1, 2, 3, 6]  # (the last output is the worst name's mean spot)
    assert np.all(np.abs(got - want)[plain] <= paid), (got - want, paid)
    # a path that ends on the other side of a barrier changes a payment by its size: within the payment's own error
    assert np.all(np.abs(got - want)[[4, 5]] <= 4 * se[[4, 5]]), (got - want, se)


@pytest.mark.parametrize("names,n_x,n_pairs", CASES)
def test_float_ladders_equal_those_of_the_pieces(names, n_x, n_pairs):
    whole, _ = result_arrays(engine.mc_price(mc_request(**_ladder(names, n_x, n_pairs)), "fp32"))
    total = np.zeros(len(whole))
    for at in range(0, n_pairs, SMALL):
        r = engine.mc_price(mc_request(**_ladder(names, n_x, min(SMALL, n_pairs - at), at)), "fp32")
        total += np.array(r.sum_y[:len(whole)])
    assert np.allclose(whole, total / n_pairs, rtol=1e-13, atol=0)  # the same pair values, in another order in FP64


@pytest.mark.parametrize("kind", [1, 0])
def test_observations_on_the_edges_of_eight_step_batches_are_all_taken(oracle, kind):
    kw = dict(_ladder(1, 120, WHOLE), kind=[kind], cvar=[0.04])
    for k in ("leg_type", "leg_strike", "leg_barrier", "leg_level", "discount"):
        del kw[k]
    steps = np.array([1, 8, 9, 16, 17, 40, 41, 42, 64, 100, 125, 126])
    kw.update(product=1, obs_step=steps, obs_discount=np.full(len(steps), 1.0),
              trigger=[1.02] * (len(steps) - 1) + [0.0], coupon_barrier=0.9, coupon=0.01, ki_barrier=0.8,
              put_strike=1.0, memory=1, ki_daily=1)
    got, _ = result_arrays(engine.mc_price(mc_request(**kw), "fp32"))
    want, se = result_arrays(oracle.mc_price(mc_request(**kw)))
    # (a date that is not observed moves the mean count of coupons, the last output, by a tenth and more)
    assert np.all(np.abs(got - want) <= 4 * se + 1e-12), (got - want, se)
    assert 4 * se[3] < 0.1
