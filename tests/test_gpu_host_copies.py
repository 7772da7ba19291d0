"""The one-shot calls' host copies at their edges: a table larger than the two pinned slots it is uploaded through, and
columns widened into an array that no 16-byte store can start on."""

import numpy as np
import pytest

from optlab_b200 import engine
from optlab_b200.requests import paths_request

pytestmark = pytest.mark.gpu


def _request(table, step_row, n_pairs, n_x, out=None):
    rows, steps = len(table), len(step_row)
    return paths_request(dt=np.full(steps, 1 / 52), t0=np.arange(steps) / 52, obs_step=np.arange(1, steps + 1),
                         root=np.eye(1), kind=[1], cvar=[0.0], heston=[0.0, 1, 1, 0, 0], same=1,
                         fwd=np.full((1, steps), 100.0), n_pairs=n_pairs, seed=5, step_row=step_row,
                         lo=np.full(rows, -0.5), inv_dx=np.full(rows, n_x - 1.0), table=table, n_x=n_x, out=out)


def _out(held):
    return next(a for a in held.keep if isinstance(a, np.ndarray) and a.ndim == 3)


@pytest.mark.parametrize("precision,rows", [("fp32", 2200), ("fp64", 1100)])
def test_a_table_beyond_both_upload_slots_arrives_whole(precision, rows):
    n_x = 4002  # an odd number of intervals: 70 MB of them, three slots' worth
    used = np.array([0, 1, rows // 2, rows - 2, rows - 1])
    table = np.full((rows, n_x), 9.0)
    table[used] = 0.04 + 0.02 * np.random.default_rng(2).random((len(used), n_x))
    whole = _request(table, used, 301, n_x)
    part = _request(table[used], np.arange(len(used)), 301, n_x)
    engine.paths(whole, precision)
    engine.paths(part, precision)
    assert np.array_equal(_out(whole), _out(part))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n_pairs", [1, 2, 65537])
def test_columns_land_in_an_array_at_an_odd_double(precision, n_pairs):
    table = np.full((3, 11), 0.04)
    held = _request(table, [0, 1, 2], n_pairs, 11)
    engine.paths(held, precision)
    buf = np.full(3 * 2 * n_pairs + 2, -7.0)
    assert buf.ctypes.data % 16 == 0
    odd = _request(table, [0, 1, 2], n_pairs, 11, out=buf[1:-1].reshape(1, 3, 2 * n_pairs))
    engine.paths(odd, precision)
    assert np.array_equal(_out(odd), _out(held)) and buf[0] == -7.0 and buf[-1] == -7.0
