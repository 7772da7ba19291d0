"""Streamed table rows, and a pair's legs on two lanes, against the same pairs priced by the other kernels (rows read from
global memory, whole pairs): they step alike, so columns and pair values agree bit for bit; sizes around the ranges'
ends, steps around a stage, row lengths of odd and even interval counts, repeated rows, several passes a block."""

import numpy as np
import pytest

from optlab_b200 import engine, workloads
from optlab_b200 import script as sc
from optlab_b200._abi import OB_MODEL_PATHS
from optlab_b200.models import correlation_root
from optlab_b200.requests import mc_request, paths_request, result_arrays

pytestmark = pytest.mark.gpu

# 148 SMs stream 16103 to 56831 pairs (one name; to 94719 in paths and scripts): the range's ends and a ragged count
STREAMED = [16103, 30001, 56831]
SMALL = 4096  # pairs read from global memory (prices: with a pair's legs on two lanes), to compare with


def _model(names, steps, n_x, n_pairs, seed=31):
    rng = np.random.default_rng(4)
    t0 = np.arange(steps) / 252.0
    rows = names * steps
    step_row = np.arange(rows).reshape(names, steps).copy()
    step_row[:, 2:5] = step_row[:, 1:2]  # a row used by several steps
    table = 0.04 * (1 + 0.2 * rng.random((rows, 1))) + 0.01 * np.linspace(1, -1, n_x)[None, :] ** 2
    corr = np.full((names, names), 0.4) + 0.6 * np.eye(names)
    return dict(dt=np.full(steps, 1 / 252), t0=t0, n_pairs=n_pairs, seed=seed, kind=[1] * names, cvar=np.zeros(names),
                root=correlation_root(corr) if names > 1 else np.eye(1), step_row=step_row, lo=np.full(rows, -0.8),
                inv_dx=np.full(rows, (n_x - 1) / 1.6), table=table, n_x=n_x)


def _out(held):
    return next(a for a in held.keep if isinstance(a, np.ndarray) and a.ndim == 3)


@pytest.mark.parametrize("n_pairs", STREAMED)
@pytest.mark.parametrize("steps,n_x", [(29, 801), (33, 800), (64, 400)])
def test_streamed_columns_equal_those_of_rows_in_global_memory(n_pairs, steps, n_x):
    obs = [0, 1, steps // 2, steps]
    kw = dict(obs_step=obs, heston=[0.0, 1, 1, 0, 0], same=1, fwd=np.full((1, len(obs)), 100.0), win_lo=[1], win_hi=[3])
    whole = paths_request(**_model(1, steps, n_x, n_pairs), **kw)
    engine.paths(whole, "fp32")
    first = paths_request(**_model(1, steps, n_x, SMALL), **kw)
    engine.paths(first, "fp32")
    last = paths_request(**_model(1, steps, n_x, SMALL), **kw, first_pair=n_pairs - SMALL)
    engine.paths(last, "fp32")
    w, f, z = _out(whole), _out(first), _out(last)
    for leg in (0, 1):
        at = leg * n_pairs
        assert np.array_equal(w[:, :, at:at + SMALL], f[:, :, leg * SMALL:(leg + 1) * SMALL])
        assert np.array_equal(w[:, :, at + n_pairs - SMALL:at + n_pairs], z[:, :, leg * SMALL:(leg + 1) * SMALL])


@pytest.mark.parametrize("n_pairs", [*STREAMED, 3 * 65536])
@pytest.mark.parametrize("names", [1, 2, 3])
@pytest.mark.parametrize("steps,n_x", [(29, 801), (57, 400), (40, 60), (8, 60), (5, 2)])
def test_prices_equal_those_of_the_pieces(names, n_pairs, steps, n_x):
    m = workloads.FlatMarket(100.0, 0.02, 0.01)
    args = _model(names, steps, n_x, n_pairs)
    t_end = np.concatenate([[0.0], args["t0"] + args["dt"]])
    obs = np.unique([steps // 3, steps // 2, steps])
    fields = dict(model=OB_MODEL_PATHS, spot=np.full(names, 100.0), log_fwd=np.tile(m.log_fwd(t_end), (names, 1)),
                  product=1, obs_step=obs, obs_discount=m.D(obs / 252), trigger=[1.0] * (len(obs) - 1) + [0.0], coupon_barrier=0.95,
                  coupon=0.02, ki_barrier=0.9, put_strike=1.0, memory=1, ki_daily=1)
    whole, _ = result_arrays(engine.mc_price(mc_request(**args, **fields), "fp32"))
    total = np.zeros(4)
    for at in range(0, n_pairs, SMALL):  # pieces below the range: legs on two lanes
        count = min(SMALL, n_pairs - at)
        piece = dict(args, n_pairs=max(count, 2), first_pair=at)
        r = engine.mc_price(mc_request(**piece, **fields), "fp32")
        if count < 2:
            pytest.skip("a piece of one pair")
        total += np.array(r.sum_y[:4])
    # the same pair values, summed in another order in FP64
    assert np.allclose(whole, total / n_pairs, rtol=1e-13, atol=0)


@pytest.mark.parametrize("n_pairs", STREAMED)
@pytest.mark.parametrize("window", ["lowest", "highest", None])
def test_a_streamed_script_equals_its_pair_values_in_pieces(n_pairs, window):
    steps = 45
    args = _model(1, steps, 801, n_pairs)
    t = steps / 252
    fix = f"{window}(X, t=0, t={t!r}, n={steps})" if window else "X"
    comp = sc.compile_script(f"underlying X\nevent t={t!r} pay t={t!r}\n  pay max({fix} / 100, 0.9) as redemption\nend\n")
    t_end = np.concatenate([[0.0], args["t0"] + args["dt"]])
    base = dict(model=OB_MODEL_PATHS, spot=[100.0], log_fwd=0.01 * t_end[None, :], product=1, obs_step=[steps],
                obs_discount=[1.0], trigger=[0.0])

    def values(count, first):
        sim = mc_request(**dict(args, n_pairs=count, first_pair=first), **base)
        held = sc.script_request(comp, sim, lambda s: 1.0, pair_values=True)
        r = sc.run(held, "fp32")
        return r, held.keep[1]["pair_value"]

    whole, v = values(n_pairs, 0)
    part, w = values(SMALL, 0)
    assert np.array_equal(v[:SMALL], w)
    assert abs(whole.price / v.mean() - 1) < 1e-12


@pytest.mark.parametrize("n_x", [2, 3, 4, 5])
def test_short_rows_of_a_large_table_equal_those_of_a_staged_one(n_x):
    # 20000 rows of one to four intervals do not fit the stage; the rows the steps read alone do
    steps, n_pairs, spare = 40, 30001, 20000
    args = _model(1, steps, n_x, n_pairs)
    kw = dict(obs_step=[steps // 2, steps], heston=[0.0, 1, 1, 0, 0], same=1, fwd=np.full((1, 2), 100.0))
    large = dict(args, step_row=args["step_row"] + spare, lo=np.full(spare + steps, -0.8),
                 inv_dx=np.full(spare + steps, (n_x - 1) / 1.6),
                 table=np.vstack([np.full((spare, n_x), 0.5), args["table"]]))
    staged, streamed = paths_request(**args, **kw), paths_request(**large, **kw)
    engine.paths(staged, "fp32"), engine.paths(streamed, "fp32")
    assert np.array_equal(_out(staged), _out(streamed))
